"""GPU: field transfers between a handle and device buffers (row copies, widening, reset).

Rows whose lengths and addresses allow chunks of 16, 8, 4 and 2 bytes, contiguous grids, and
buffers that a kernel on the handle's device may not touch (pinned host memory) give the same
bytes; reset clears fields, DFT sums and CPML psi and a second run repeats the first.
"""
import numpy as np
import pytest

import gdiamond_b200 as gd
from gdiamond_b200 import workloads as W

pytestmark = pytest.mark.gpu

DTYPE = {"f32": [np.float32] * 6, "f16": [np.float16] * 6, "f64": [np.float64] * 6,
         "f16e": [np.float16] * 3 + [np.float32] * 3}


@pytest.mark.parametrize("storage", ["f32", "f16", "f16e", "f64"])
@pytest.mark.parametrize("shape", [(32, 5, 7), (33, 4, 6), (34, 7, 3), (36, 3, 5), (250, 3, 4),
                                   (3, 3, 3), (1030, 3, 3)])
def test_planes_roundtrip_and_widened_reads(shape, storage):
    import torch
    nx, ny, nz = shape
    rng = np.random.default_rng(nx)
    sim = gd.Simulation(*shape, storage=storage)
    if storage in ("f16", "f16e"):
        sim.set_storage_scale([4.0, 1.0, 0.5, 1.0, 2.0, 1.0])
    for c in range(6):
        dt = DTYPE[storage][c]
        a = rng.normal(size=(nz, ny, nx)).astype(dt)
        raw = torch.from_numpy(a.view(np.uint8).reshape(-1).copy())
        for off in (0, dt().itemsize):  # a buffer that starts on one element's boundary only
            buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda")
            buf[off:off + raw.numel()] = raw.cuda()
            torch.cuda.synchronize()
            sim.set_planes_device(c, 0, nz, buf.data_ptr() + off)
            back = torch.full_like(buf, 7)
            torch.cuda.synchronize()
            sim.get_planes_device(c, 1, nz - 1, back.data_ptr() + off)
            sim.sync()
            n = a[1:].nbytes
            assert bytes(back[off:off + n].cpu().numpy()) == a[1:].tobytes()
            assert (back[off + n:].cpu().numpy() == 7).all() and (back[:off].cpu().numpy() == 7).all()
        scale = np.float32(sim.storage_scale[c]) if dt == np.float16 else np.float32(1)
        want = a.astype(np.float32) * scale
        out = torch.full((nz * ny * nx + 8,), -1.0, device="cuda")
        pinned = torch.full((nz * ny * nx,), -1.0).pin_memory()
        torch.cuda.synchronize()
        sim.get_field_device(c, out.data_ptr())
        sim.get_field_device(c, pinned.data_ptr())
        sim.sync()
        assert np.array_equal(out[:want.size].cpu().numpy(), want.reshape(-1))
        assert (out[want.size:].cpu().numpy() == -1.0).all()
        assert np.array_equal(pinned.numpy(), want.reshape(-1))
        assert np.array_equal(sim.get_field(c), want.reshape(-1))
    sim.close()


@pytest.mark.parametrize("cpml", [False, True])
def test_reset_clears_everything_a_run_reads(cpml):
    shape = (37, 30, 26)
    sim = gd.Simulation(*shape)
    sim.set_coefficients(W.vacuum_coefficients(shape))
    if cpml:
        sim.set_cpml(thickness=5)
    sim.set_sources([dict(component="Jz", wave=W.gaussian_wave(40, delay=5.0), i=18, j=15, k=13)])
    f = W.source_band(5)
    fid = sim.add_flux_monitor(12, f)
    mids = [sim.add_dft_monitor("Ez", 4, f) for _ in range(6)]
    runs = []
    for T in (20, 21, 20):
        sim.reset()
        assert sim.t == 0 and all(not a.any() for a in sim.fields())
        assert all(not a.any() for m in mids for a in sim.get_dft(m))
        if cpml:
            assert all(not p.any() for p in sim.cpml_state())
        sim.step(T)
        runs.append([sim.get_flux(fid)] + sim.fields() + [a for m in mids for a in sim.get_dft(m)])
    assert runs[0][0].any() and all(np.array_equal(a, b) for a, b in zip(runs[0], runs[2]))
    sim.close()
