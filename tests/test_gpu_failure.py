"""GPU failure detection without a GPU fault: a bounded wait that runs out.

The reference's error path is CUDACHECK -> printf + exit(1) (gDiamond/gdiamond_gpu.cuh:11-20).
Here every mbarrier wait of the tiled kernels is bounded; when one gives up, the tile records
FDTD_ERR_DEVICE_TIMEOUT in the handle's device error word, waits (bounded) for its own copies in
flight, and leaves its z-march; fdtd_sync reports the status.  The test hook
fdtd_debug_fail_copy makes one tile skip issuing one plane copy, so its wait has nothing to
wait for (a flag that nothing sets) and runs out after a short limit.  Nothing faults, traps or
hangs: the context stays usable, which the test shows by resetting and stepping bit-exactly
against the oracle afterwards.
"""
import numpy as np
import pytest

import oracle
import gdiamond_b200 as gd
from gdiamond_b200 import workloads as W
from test_gpu_parity import assert_fields_match, osrc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,blt,rows,storage", [("tiled_w32p", 2, 24, "f32"),
                                                     ("tiled_w64", 3, 16, "f32"),
                                                     ("tiled_w32p", 2, 32, "f16e")])
def test_expired_wait_reports_timeout_and_handle_recovers(family, blt, rows, storage):
    shape, T = (70, 52, 41), 12
    coefs = W.reference_coefficients(shape)
    w = W.gaussian_wave(T, delay=4.0, width=2.0, period=5.0)
    src = [dict(component="Jz", wave=w, i=35, j=26, k=20)]
    sim = gd.Simulation(*shape, kernel=family, blt=blt, tile_rows=rows, z_chunks=2,
                        storage=storage)
    sim.set_coefficients(coefs)
    sim.set_sources(src)
    sim.step(blt)  # tunes nothing (one configuration) and runs cleanly
    sim.sync()
    sim.debug_fail_copy((1, 1, 0), iteration=5, wait_cycles=2_000_000)  # ~1 ms
    sim.step(blt)
    with pytest.raises(gd.FdtdError) as e:
        sim.sync()
    assert e.value.status == 5  # FDTD_ERR_DEVICE_TIMEOUT
    sim.sync()  # reported once, then cleared
    # the hook fired once; after a reset the handle steps correctly
    sim.reset()
    sim.step(T)
    sim.sync()
    if storage == "f32":
        F_ref = oracle.run(shape, coefs, T, sources=[osrc(s) for s in src])
        assert_fields_match(sim.fields(), F_ref, f"after timeout {family}")
    else:
        assert all(np.isfinite(f).all() for f in sim.fields())
    sim.close()


_RESET = """
import ctypes, sys
import numpy as np
import gdiamond_b200 as gd
from gdiamond_b200 import workloads as W

def work():
    out = []
    shape = (70, 52, 41)
    for kernel, rows in (("tiled_w32", 16), ("tiled_w64", 16), ("tiled_w32p", 32)):
        sim = gd.Simulation(*shape, kernel=kernel, blt=2, tile_rows=rows, z_chunks=2, min_blocks=1)
        sim.set_coefficients(W.vacuum_coefficients(shape))
        sim.set_sources([dict(component="Jz", wave=W.gaussian_wave(8, delay=3.0), i=35, j=26, k=20)])
        if kernel == "tiled_w32p":
            b = gd.Batch([sim])
            b.step(5)  # the last step's instance is first launched while the graph is captured
            b.close()
        sim.step(4)
        sim.sync()
        out += sim.fields()
        sim.close()
    rng = np.random.default_rng(0)
    x, y = rng.normal(size=(2048, 6)).astype(np.float32), rng.normal(size=(2048, 32)).astype(np.float32)
    for members in (2, 5):
        net = gd.MLP((6, 64, 32), members=members, seed=1)
        net.set_data(x, y)
        net.train(1, batch=64)
        out += [net.get_params()] + list(net.predict(x)) + [net.grad(x, y)[1]]
        net.close()
    return out

first = work()
rt = ctypes.CDLL([l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l][0])
assert rt.cudaDeviceSynchronize() == 0 and rt.cudaDeviceReset() == 0
for a, b in zip(first, work()):
    assert np.array_equal(a, b) or np.allclose(a, b, rtol=1e-4, atol=1e-6)
print("same after the reset")
"""


def test_new_handles_work_after_a_device_reset():
    """cudaDeviceReset ends the process's context and with it every kernel attribute that was
    set; handles made afterwards run as the first ones did."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _RESET], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "same after the reset" in r.stdout, r.stderr[-2000:]
