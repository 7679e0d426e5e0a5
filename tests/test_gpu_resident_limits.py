"""The state-on-chip kernel (k_resident) at the limits of what it takes."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402
from strata_fdtd_gb300 import _native  # noqa: E402

from test_gpu_pipe import _check  # noqa: E402
from test_gpu_resident import _fill, _resident  # noqa: E402


@pytest.mark.parametrize("shape,stretched,on_chip", [
    ((1000, 1, 1000), False, True), ((1200, 1, 1200), False, True), ((3000, 1, 400), False, True),
    ((800, 2, 1000), False, True), ((1, 900, 1100), False, False), ((1000, 1000, 1), False, False),
    ((1, 250, 1100), False, True), ((900, 500, 1), False, True), ((800, 2, 1000), True, True),
    ((2, 700, 900), True, False)])
def test_thin_grids_equal_single_steps(shape, stretched, on_chip):
    """Grids of one or two cells along an axis, up to 1.4 million cells: whole blocks
    have no neighbour along it.  (One cell along x leaves a thread one plane, one along z
    a quarter of its cells: fewer fit on the chip.)"""
    out = []
    rng = np.random.default_rng(shape[0])
    coords = [np.cumsum(rng.uniform(0.7, 1.4, n)) * 1e-3 for n in shape]
    for single in (False, True):
        if stretched:
            s = S.FDTDSolver(grid=S.NonuniformGrid(*coords), c=343.0, rho=1.2, courant=0.6)
        else:
            s = S.FDTDSolver(shape=shape, resolution=1e-3, c=343.0, rho=1.2, courant=0.6)
        mask = np.ones(shape, bool)
        mask[tuple(slice(n // 3, n // 3 + 40) if n > 2 else slice(0, 1) for n in shape)] = False
        s.set_geometry(mask)
        s.add_source(S.GaussianPulse(position=tuple(n // 2 for n in shape), frequency=20000.0))
        s.add_probe("a", tuple(n - 1 for n in shape))
        if single:
            s.set_kernel("tile1_r2_w8")
        out.append(s)
    _fill(*out, 3)
    assert _resident(out[0], 9) == on_chip
    for n in (9, 14):
        for s in out:
            s.run_steps(n)
    _check(*out, shape)


@pytest.mark.parametrize("read", ["microphone", "field", "async", "energy"])
def test_an_expired_wait_is_seen_by_every_read(read):
    """The bounded wait's test hook on a solver with a microphone and no probe: what is
    read first raises, so does what is read after it, and a run from a reset is exact."""
    def build():
        s = S.FDTDSolver(shape=(40, 41, 44), resolution=1e-3, c=343.0, rho=1.2, courant=0.6)
        s.add_source(S.GaussianPulse(position=(20, 20, 20), frequency=20000.0))
        s.add_microphone(position=(0.021, 0.019, 0.022), name="m")
        return s

    reads = {"microphone": lambda s: s.microphones["m"].get_waveform(), "field": lambda s: s.p,
             "async": lambda s: s.fields_async(("p",))(), "energy": lambda s: s.compute_energy()}
    s, ref = build(), build()
    lib = _native.load()
    _native.check(lib.sf_plan_set_wait_limit(s._plan, 2000, 1), "sf_plan_set_wait_limit")
    s.run_steps(10)
    for q in [read] + sorted(reads):
        with pytest.raises(_native.NativeError, match="dependency wait expired"):
            reads[q](s)
    _native.check(lib.sf_plan_set_wait_limit(s._plan, 0, 0), "sf_plan_set_wait_limit")
    s.reset()
    for q in ("p", "vx", "vy", "vz"):
        assert not getattr(s, q).any()
    s.run_steps(10)
    ref.run_steps(10)
    _check(s, ref, read)
    np.testing.assert_array_equal(reads["microphone"](s), reads["microphone"](ref))


def test_an_expired_wait_is_seen_by_the_energy_reading_without_allocations():
    s = S.FDTDSolver(shape=(40, 41, 44), resolution=1e-3, c=343.0, rho=1.2, courant=0.6)
    s.add_source(S.GaussianPulse(position=(20, 20, 20), frequency=20000.0))
    lib = _native.load()
    out = ctypes.c_double()

    def energy():
        return lib.sf_plan_energy_noalloc(s._plan, s.rho, s.c, s.dx, ctypes.byref(out), s._stream())

    s.run_steps(10)
    assert energy() == 0 and out.value > 0
    _native.check(lib.sf_plan_set_wait_limit(s._plan, 2000, 1), "sf_plan_set_wait_limit")
    s.run_steps(10)
    assert energy() != 0 and b"wait expired" in lib.sf_last_error()
    assert energy() == 0  # (reported once)


def test_buffers_are_released_behind_a_run_in_flight():
    """sf_release_deferred() while the state-on-chip kernel runs: it waits for the run,
    and leaves no error behind for the next launch."""
    lib = _native.load()

    def build(kernel=None):
        s = S.FDTDSolver(shape=(96, 92, 100), resolution=1e-3, c=343.0, rho=1.2, courant=0.6)
        s.add_source(S.GaussianPulse(position=(40, 41, 42), frequency=20000.0))
        s.add_probe("a", (50, 50, 50))
        if kernel:
            s.set_kernel(kernel)
        return s

    a, b, c, ref = build(), build("col4"), build(), build("col4")
    assert _resident(a, 40000)
    for s in (b, ref):
        s.run_steps(1)
    a.run_steps(9)
    torch.cuda.synchronize()
    _native.check(lib.sf_release_deferred())  # (nothing else is queued for release)
    a.run_steps(9)
    a.run_steps(40000)  # about 0.16 s
    _native.check(lib.sf_release_deferred())
    assert torch.cuda.current_stream().query()
    b.run_steps(8)
    ref.run_steps(8)
    c.run_steps(9)  # new mailboxes
    _check(b, ref, "behind the release")
    _check(c, ref, "new mailboxes")
    a.synchronize()


@pytest.mark.parametrize("shape", [(40, 41, 44), (96, 92, 100)])
def test_the_tuner_times_the_state_on_chip_kernel(shape):
    """It is the faster one on these grids and keeps its calls; the trials leave the
    state alone, with an odd number of steps behind it too."""
    out = []
    for tune in (False, True):
        s = S.FDTDSolver(shape=shape, resolution=1e-3, c=343.0, rho=1.2, courant=0.6)
        s.add_boundary(S.ABCFirstOrder())
        s.add_source(S.GaussianPulse(position=(20, 20, 20), frequency=20000.0))
        s.add_probe("a", (30, 30, 30))
        s.run_steps(11)
        if tune:
            s.autotune(launches=3)
        assert _resident(s, 40)
        s.run_steps(9)
        out.append(s)
    _check(*out, shape)
