"""The surrogate's GPU MLP ensemble (fdtd_mlp_*) against the CPU FP64 oracle (oracle/mlp.py).

* gradients of every member (BF16 tensor-core GEMMs, FP32 accumulation) against the oracle
  with the same BF16 roundings (tight) and against exact FP64 backprop (loose), for both GEMM
  paths (tcgen05 with a TMEM accumulator, and warp-level mma.sync), and the two paths against
  each other on odd shapes;
* forward outputs of every member and the ensemble mean / standard deviation;
* one Adam step against the oracle's Adam on the oracle's gradient;
* training on a smooth function lowers the loss and generalises; invalid arguments fail.
"""
import numpy as np
import pytest

import gdiamond_b200 as gd
from oracle import mlp as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def data(n, dims, seed):
    rng = np.random.default_rng(seed)
    return (rng.uniform(-1, 1, (n, dims[0])).astype(np.float32),
            rng.normal(0, 1, (n, dims[-1])).astype(np.float32))


@pytest.mark.parametrize("dims,members,n", [((6, 37, 19, 3), 2, 70), ((7, 200, 130, 72), 3, 333),
                                            ((6, 256, 256, 256, 64), 4, 1000)])
def test_gemm_paths_agree(dims, members, n):
    x, y = data(n, dims, 9)
    out = {}
    for gemm in ("mma_sync", "tcgen05"):
        net = gd.MLP(dims, members=members, seed=5, gemm=gemm)
        mean, sd, per = net.predict(x, members=True)
        loss, g = net.grad(x, y)
        out[gemm] = (per, loss, g)
        net.close()
    (p0, l0, g0), (p1, l1, g1) = out["mma_sync"], out["tcgen05"]
    assert rel(p1, p0) <= 1e-4, rel(p1, p0)
    assert np.allclose(l1, l0, rtol=1e-4)
    for e in range(members):
        assert rel(g1[e], g0[e]) <= 2e-3, (e, rel(g1[e], g0[e]))


@pytest.mark.parametrize("gemm", ["tcgen05", "mma_sync"])
@pytest.mark.parametrize("dims,members,n", [((6, 256, 256, 256, 64), 4, 200),
                                            ((5, 37, 19, 3), 2, 70)])
def test_gradients_match_oracle(dims, members, n, gemm):
    net = gd.MLP(dims, members=members, seed=7, gemm=gemm)
    x, y = data(n, dims, 1)
    loss, g = net.grad(x, y)
    P = net.get_params()
    for e in range(members):
        L = [(W.astype(np.float64), b.astype(np.float64)) for W, b in net.unpack(P[e])]
        lq, gq = O.loss_and_grad(L, x, y, bf16=True)
        lx, gx = O.loss_and_grad(L, x, y, bf16=False)
        assert abs(loss[e] - lq) <= 1e-4 * lq
        assert abs(loss[e] - lx) <= 2e-2 * lx
        got = net.unpack(g[e])
        for n_, ((dW, db), (qW, qb), (xW, xb)) in enumerate(zip(got, gq, gx)):
            assert rel(dW, qW) <= 2e-3, (e, n_, "W", rel(dW, qW))
            assert rel(db, qb) <= 2e-3, (e, n_, "b", rel(db, qb))
            assert rel(dW, xW) <= 5e-2, (e, n_, "W exact", rel(dW, xW))
            assert rel(db, xb) <= 5e-2, (e, n_, "b exact", rel(db, xb))
    net.close()


@pytest.mark.parametrize("gemm", ["tcgen05", "mma_sync"])
def test_forward_and_ensemble_statistics_match_oracle(gemm):
    dims = (6, 256, 256, 256, 64)
    net = gd.MLP(dims, members=4, seed=3, gemm=gemm)
    x, _ = data(333, dims, 2)
    mean, sd, per = net.predict(x, members=True)
    P = net.get_params()
    outs = []
    for e in range(4):
        L = [(W.astype(np.float64), b.astype(np.float64)) for W, b in net.unpack(P[e])]
        ref, _ = O.forward(L, x, bf16=True)
        assert rel(per[e], ref) <= 1e-3, (e, rel(per[e], ref))
        outs.append(per[e].astype(np.float64))
    outs = np.array(outs)
    assert np.allclose(mean, outs.mean(0), rtol=1e-5, atol=1e-5)
    assert np.allclose(sd, outs.std(0), rtol=1e-4, atol=1e-5)
    assert sd.mean() > 0  # members start from different seeds
    net.close()


def test_layout_and_param_roundtrip():
    dims = (6, 256, 256, 256, 64)
    net = gd.MLP(dims, members=2, seed=0)
    for w, (o, i), b in net.layout():
        assert w % 8 == 0 and b % 8 == 0 and b >= w + o * i
    assert net.n_params >= sum(o * i + o for _, (o, i), _ in net.layout())
    P = net.get_params()
    P2 = P * np.float32(0.5)
    net.set_params(P2)
    assert np.array_equal(net.get_params(), P2)
    net.close()


def test_first_adam_step_matches_oracle():
    dims = (6, 64, 64, 8)
    net = gd.MLP(dims, members=2, seed=11)
    x, y = data(96, dims, 4)
    P0 = net.get_params()
    net.set_data(x, y)
    net.train(epochs=1, batch=96, lr=1e-3, seed=0)  # one full-batch step per member
    P1 = net.get_params()
    for e in range(2):
        L = [(W.astype(np.float64), b.astype(np.float64)) for W, b in net.unpack(P0[e])]
        _, gq = O.loss_and_grad(L, x, y, bf16=True)
        flat = np.zeros(net.n_params)
        for (w, (o, i), b), (dW, db) in zip(net.layout(), gq):
            flat[w:w + o * i] = dW.reshape(-1)
            flat[b:b + o] = db
        want, _, _ = O.adam(P0[e].astype(np.float64), flat, 0.0, 0.0, t=1, lr=1e-3)
        used = np.zeros(net.n_params, bool)
        for w, (o, i), b in net.layout():
            used[w:w + o * i] = True
            used[b:b + o] = True
        d_got = (P1[e] - P0[e])[used].astype(np.float64)
        d_want = (want - P0[e])[used]
        # the first Adam step moves every parameter by ~lr * sign(gradient)
        close = np.abs(d_got - d_want) <= 2e-6 + 1e-3 * np.abs(d_want)
        assert close.mean() >= 0.99, close.mean()
        assert np.array_equal(P1[e][~used], P0[e][~used])
    net.close()


def test_training_fits_a_smooth_function():
    dims = (6, 256, 256, 256, 64)
    rng = np.random.default_rng(0)
    A = rng.normal(0, 1, (6, 64))
    f = lambda x: np.sin(x @ A * 0.7) + 0.3 * np.cos(x @ A * 0.3)  # noqa: E731
    x = rng.uniform(-1, 1, (2048, 6)).astype(np.float32)
    xt = rng.uniform(-1, 1, (256, 6)).astype(np.float32)
    net = gd.MLP(dims, members=4, seed=1)
    net.set_data(x, f(x))
    losses = net.train(epochs=60, batch=64, lr=1e-3, seed=2)
    assert losses.shape == (60, 4) and np.all(np.isfinite(losses))
    assert np.all(losses[-1] < 0.05 * losses[0])
    mean, sd = net.predict(xt)
    err = rel(mean, f(xt))
    assert err < 0.1, err
    # the ensemble spread tracks the error: larger off the training range
    _, sd_far = net.predict(xt * 3)
    assert sd_far.mean() > sd.mean()
    net.close()


def test_invalid_arguments():
    with pytest.raises(gd.FdtdError):
        gd.MLP((6,), members=1)
    with pytest.raises(gd.FdtdError):
        gd.MLP((6, 0, 4), members=1)
    net = gd.MLP((4, 8, 2), members=1)
    with pytest.raises(gd.FdtdError):
        net.train(epochs=1)  # no data
    with pytest.raises(KeyError):
        net.set_gemm("wmma")
    with pytest.raises(ValueError):
        net.set_data(np.zeros((3, 4)), np.zeros((2, 2)))
    net.close()


@pytest.mark.parametrize("n", [1, 127, 129, 70000])
def test_fused_inference_matches_layer_by_layer(n):
    """predict() on the tcgen05 path runs every layer in one kernel (activations kept in shared
    memory); the warp-level path runs the layers one GEMM at a time."""
    dims = (6, 256, 256, 256, 64)
    x, _ = data(n, dims, 11)
    out = {}
    for gemm in ("tcgen05", "mma_sync"):
        net = gd.MLP(dims, members=4, seed=8, gemm=gemm)
        out[gemm] = net.predict(x, members=True)
        net.close()
    (m1, s1, p1), (m0, s0, p0) = out["tcgen05"], out["mma_sync"]
    assert np.all(np.isfinite(p1))
    assert rel(p1, p0) <= 1e-3, rel(p1, p0)
    assert rel(m1, m0) <= 1e-3


# Slices of 1 and 2 column groups and idle CTAs (widths 16..256), partial row tiles, a short last
# batch, one row, the largest batch, odd input widths, one hidden layer and eight layers.
@pytest.mark.parametrize("dims,members,n,batch", [
    ((6, 256, 256, 256, 64), 4, 300, 64), ((6, 96, 64), 1, 130, 100), ((7, 16, 16), 2, 65, 64),
    ((1, 48, 128, 32), 3, 129, 128), ((64, 240, 16), 2, 77, 33), ((5, 32, 16, 48), 1, 5, 1),
    ((6,) + (32,) * 8, 2, 90, 48), ((6, 256, 144, 64), 5, 200, 128)])
def test_fused_training_epoch_equals_separate_launches(dims, members, n, batch):
    """The one-launch epoch runs the products, sums and updates of the launch-per-product path in
    the same order: parameters after three epochs are equal bit for bit (the summed losses are
    accumulated with atomics: relative 1e-5)."""
    x, y = data(n, dims, 3)
    out = {}
    for gemm in ("mma_sync", "auto"):
        net = gd.MLP(dims, members=members, seed=11, gemm=gemm)
        net.set_data(x, y)
        loss = np.concatenate([net.train(2, batch=batch, lr=1e-3, seed=4),
                               net.train(1, batch=batch, lr=3e-4, seed=5)])
        out[gemm] = (net.get_params(), loss)
        net.close()
    assert np.array_equal(out["auto"][0], out["mma_sync"][0])
    assert np.allclose(out["auto"][1], out["mma_sync"][1], rtol=1e-5)


# Widths that are no multiple of the 64-wide K chunk: the fused kernel's activation tile is not
# cleared behind them.  Another network's activations (or NaN) are left in shared memory first.
@pytest.mark.parametrize("dims", [(6, 96, 32), (6, 160, 96, 64), (5, 32, 224, 32), (64, 96, 96, 96, 32)])
def test_fused_inference_of_widths_between_chunks(dims):
    x, _ = data(700, dims, 2)
    wide = gd.MLP((6, 256, 256, 64), members=2, seed=9)
    P = wide.get_params()
    P[:] = np.inf  # its activations become infinite and NaN
    wide.set_params(P)
    net = gd.MLP(dims, members=3, seed=4)
    ref = gd.MLP(dims, members=3, seed=4, gemm="mma_sync")
    ref.set_params(net.get_params())
    want = ref.predict(x, members=True)
    for _ in range(3):
        wide.predict(data(60000, wide.dims, 1)[0])
        got = net.predict(x, members=True)
        for a, b in zip(got, want):
            assert np.isfinite(a).all() and rel(a, b) <= 1e-3
    for n in (wide, net, ref):
        n.close()


def test_training_workspace_does_not_grow_with_an_earlier_prediction():
    """The one-launch epoch holds gradients of at most 128 rows a member, whatever number of rows
    an earlier call of the layer-by-layer path sized its own workspace for."""
    import torch
    dims, members = (6, 144, 144, 48), 16
    x, y = data(65536, dims, 1)
    net = gd.MLP(dims, members=members, seed=2)
    net.predict(x)  # widths that are no multiples of 32: a layer at a time
    net.set_data(x[:500], y[:500])
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    net.train(1, batch=64)
    used = before - torch.cuda.mem_get_info()[0]
    net.close()
    # gradients: 16 members x 128 rows x 336 columns x 2 bytes = 1.4 MB; allocations of 2 MB each
    assert used <= 32 << 20, used


def test_training_without_room_for_the_epoch_workspace():
    """When the one-launch epoch's gradients cannot be allocated, the separate launches, which need
    no more memory than they hold, train the same parameters."""
    import ctypes
    import torch
    dims, members = (6, 256, 256, 256, 64), 64  # gradients: 4 MB a hidden layer
    x, y = data(200, dims, 3)
    want = gd.MLP(dims, members=members, seed=6, gemm="mma_sync")
    net = gd.MLP(dims, members=members, seed=6, gemm="mma_sync")
    for m in (want, net):
        m.set_data(x, y)
        m.train(1, batch=128, lr=1e-3, seed=3)
    net.set_gemm("auto")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rt = ctypes.CDLL([q.split()[-1] for q in open("/proc/self/maps") if "libcudart.so" in q][0])
    hold = []
    for size in (1 << 30, 1 << 26, 1 << 21):  # allocations are made of 2 MB pages
        p = ctypes.c_void_p()
        while rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
            hold.append(p)
            p = ctypes.c_void_p()
        rt.cudaGetLastError()
    try:
        net.train(1, batch=128, lr=1e-3, seed=4)
    finally:
        for p in hold:
            rt.cudaFree(p)
    want.train(1, batch=128, lr=1e-3, seed=4)
    assert np.array_equal(net.get_params(), want.get_params())
    want.close()
    net.close()


def test_fused_inference_over_more_rows_than_a_chunk():
    """262144 rows and 129 more (the second chunk's offsets and short copies), then a few rows in
    the same workspace, against the layer-by-layer path."""
    dims = (6, 32, 32)
    nets = [gd.MLP(dims, members=2, seed=3, gemm=g) for g in ("auto", "mma_sync")]
    for n in (262144 + 129, 200):
        x, _ = data(n, dims, n & 15)
        got, want = (net.predict(x, members=True) for net in nets)
        for a, b in zip(got, want):
            assert a.shape == b.shape and rel(a, b) <= 1e-3
            assert rel(a[..., -129:, :], b[..., -129:, :]) <= 1e-3
    for net in nets:
        net.close()


@pytest.mark.parametrize("members", [15, 16, 45, 46, 60, 61])
def test_training_of_large_ensembles_equals_separate_launches(members):
    """Ensembles whose clusters take turns, on either side of the sizes that go to the separate
    launches: parameters equal bit for bit."""
    for dims in ((6, 32, 16), (6, 32, 32, 16)):
        x, y = data(70, dims, members)
        got = []
        for gemm in ("auto", "mma_sync"):
            net = gd.MLP(dims, members=members, seed=2, gemm=gemm)
            net.set_data(x, y)
            net.train(2, batch=32, lr=1e-3, seed=1)
            got.append(net.get_params())
            net.close()
        assert np.array_equal(*got), dims
