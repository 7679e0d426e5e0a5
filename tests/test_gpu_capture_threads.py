"""Calls from one thread while another captures a graph in the global mode: a stream
capture forbids "potentially unsafe" calls (cudaMalloc among them) in every thread, so
a call that has to allocate does so in the relaxed mode."""
import ctypes
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402
from strata_fdtd_gb300 import _native  # noqa: E402


def _beside_a_capture(call):
    """call() in a thread, during this thread's capture of a graph; its result or
    exception, and whether the captured graph works."""
    x = torch.zeros(1000, device="cuda")
    out = []

    def run():
        try:
            out.append(call())
        except Exception as e:  # noqa: BLE001 - looked at below
            out.append(e)

    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        x.add_(1.0)
        t = threading.Thread(target=run)
        t.start()
        t.join()
        x.add_(1.0)
    g.replay()
    assert float(x.sum()) == 2000.0
    return out[0]


def test_first_state_on_chip_steps_beside_a_capture():
    def build():
        s = S.FDTDSolver(shape=(40, 41, 44), resolution=1e-3, c=343.0, rho=1.2, courant=0.6)
        s.add_source(S.GaussianPulse(position=(20, 20, 20), frequency=20000.0))
        s.step()
        return s

    lib = _native.load()
    s, ref = build(), build()
    src = s.source_table(24)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    _native.check(lib.sf_release_deferred())  # (the mailboxes of earlier tests)
    rc = _beside_a_capture(lambda: lib.sf_plan_step(s._plan, 24, src.data_ptr(), None,
                                                    stream.cuda_stream))
    assert rc == 0, rc
    torch.cuda.synchronize()
    ref.run_steps(24)
    s._mark_device_newer()
    for f in ("p", "vx", "vy", "vz"):
        np.testing.assert_array_equal(getattr(s, f), getattr(ref, f), err_msg=f)


def test_first_mask_beside_a_capture():
    lib = _native.load()
    ball = S.Sphere(center=(0.02, 0.02, 0.02), radius=0.013)
    prog, n = ball.program()
    shape = (40, 40, 40)
    out = torch.zeros(shape, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    _native.check(lib.sf_release_deferred())
    torch.cuda.synchronize()
    rc = _beside_a_capture(lambda: lib.sf_voxelize(
        ctypes.addressof(prog), n, *shape, 1e-3, 0, out.data_ptr(), stream.cuda_stream))
    assert rc == 0, rc
    c = (np.arange(40) + 0.5) * 1e-3
    r2 = sum((v - 0.02) ** 2 for v in np.meshgrid(c, c, c, indexing="ij"))
    got = out.cpu().numpy().astype(bool)
    clear = np.abs(np.sqrt(r2) - 0.013) > 1e-9
    np.testing.assert_array_equal(got[clear], (r2 <= 0.013 ** 2)[clear])
