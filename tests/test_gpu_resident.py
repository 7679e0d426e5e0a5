"""The state-on-chip kernel (k_resident): many steps of a small grid in one
launch, against the CPU oracle, bit for bit.

Covered: each planes-per-thread kind at the edges of its range, cuts along
one, two and three axes, partial chunks and quads at the grid's high ends,
walls across block faces, every source kind on block edges, probes, nonzero
last-plane velocities, uniform and stretched grids, odd and even step
counts, two solvers on two streams, and a wait that runs out.
"""
import numpy as np
import pytest

import cases as C

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402
from strata_fdtd_gb300 import _native  # noqa: E402
from oracle import oracle as O  # noqa: E402

from test_gpu_parity import API  # noqa: E402
from test_gpu_pipe import _case, _check  # noqa: E402

ORACLE = O.make_api()
FIELDS = ("p", "vx", "vy", "vz")


def _pair(shape, geometry=True):
    """The same solve on the GPU and on the oracle; random 2-cell walls."""
    case = _case(shape, 0, geometry=False)
    out = [C.build_case(api, case) for api in (API, ORACLE)]
    if geometry:
        rng = np.random.default_rng(sum(shape))
        small = tuple((n + 1) // 2 for n in shape)
        mask = np.kron(rng.random(small) > 0.15, np.ones((2, 2, 2)))
        mask = mask[tuple(slice(n) for n in shape)].astype(bool)
        for s in out:
            s.set_geometry(mask.copy())
    return out


def _resident(s, n):
    s._sync_tables()
    return bool(_native.load().sf_plan_resident(s._plan, n, 0, s._stream()))


def _fill(a, b, seed):
    """The same random state in both solvers, the last planes' faces included."""
    rng = np.random.default_rng(seed)
    for f in FIELDS:
        v = (rng.standard_normal(a.shape) * 1e-2).astype(np.float32)
        if f == "p":
            v[~a.geometry] = 0.0
        setattr(a, f, v.copy())
        setattr(b, f, v.copy())


@pytest.mark.parametrize("geometry", [False, True])
@pytest.mark.parametrize("shape", [
    (8, 8, 8), (9, 7, 5), (3, 40, 41), (160, 9, 6), (6, 170, 7), (7, 6, 610), (33, 35, 37),
    (52, 44, 48), (73, 72, 73), (75, 72, 77), (91, 90, 93), (93, 93, 95), (107, 106, 107),
    (109, 108, 106)])
def test_against_oracle(shape, geometry):
    s, ref = _pair(shape, geometry)
    _fill(s, ref, sum(shape))
    assert _resident(s, 9)
    for n in (9, 12):
        s.run_steps(n)
        ref.run_steps(n)
    _check(s, ref, shape)


@pytest.mark.parametrize("shape", [(144, 120, 132), (131, 129, 127), (136, 135, 133), (131, 131, 131)])
def test_largest_grids_against_single_steps(shape):
    """Two million cells (8 planes per thread) against the per-step kernels;
    a grid too large to fit takes those by itself."""
    case = _case(shape, 0)
    a, b = C.build_case(API, case), C.build_case(API, case)
    _fill(a, b, 5)
    b.set_kernel("tile1_r2_w8")
    assert not _resident(b, 20)
    a.run_steps(21)
    b.run_steps(21)
    _check(a, b, shape)


@pytest.mark.parametrize("shape", [(24, 26, 27), (64, 60, 66), (110, 64, 61)])
def test_stretched_grid_against_oracle(shape):
    rng = np.random.default_rng(shape[0])
    coords = [np.cumsum(rng.uniform(0.7, 1.4, n)) * 1e-3 for n in shape]
    out = []
    for api in (API, ORACLE):
        s = api.FDTDSolver(grid=api.NonuniformGrid(*coords), c=343.0, rho=1.2, courant=0.6)
        s.add_boundary(api.PML(depth=4))
        mask = np.ones(shape, dtype=bool)
        mask[5:11, 6:20, 3:9] = False
        s.set_geometry(mask)
        s.add_source(api.GaussianPulse(position=(12, 12, 12), frequency=20000.0))
        s.add_probe("a", (shape[0] - 1, 3, shape[2] - 1))
        out.append(s)
    s, ref = out
    _fill(s, ref, 1)
    assert _resident(s, 15)
    s.run_steps(15)
    ref.run_steps(15)
    _check(s, ref, shape)


def test_two_streams_and_a_captured_call():
    """Launches of two solvers on two streams are ordered; a call inside a
    caller's stream capture takes the single-step kernels."""
    case = _case((40, 41, 44), 0)
    a, b, ref = (C.build_case(x, case) for x in (API, API, ORACLE))
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, st in zip((a, b), streams):
            with torch.cuda.stream(st):
                s.run_steps(20)
    torch.cuda.synchronize()
    ref.run_steps(80)
    _check(a, ref, "stream 0")
    _check(b, ref, "stream 1")
    with torch.cuda.stream(streams[0]):
        g = torch.cuda.CUDAGraph()
        streams[0].synchronize()
        with torch.cuda.graph(g, stream=streams[0]):
            assert not _resident(a, 50)


def test_expired_wait_is_reported_and_the_next_run_is_exact():
    """With a bound of 2000 polls and the hook that makes block 0 wait for
    tags that nothing sends, every wait runs out: the launch ends, the next
    read reports it once, and a run from the restored state is exact."""
    case = _case((40, 41, 44), 0)
    s, ref = C.build_case(API, case), C.build_case(ORACLE, case)
    s.run_steps(10)
    ref.run_steps(10)
    saved = {f: getattr(s, f).copy() for f in FIELDS}
    lib = _native.load()
    _native.check(lib.sf_plan_set_wait_limit(s._plan, 2000, 1), "sf_plan_set_wait_limit")
    s.run_steps(10)
    with pytest.raises(_native.NativeError, match="dependency wait expired"):
        s.synchronize()
    _native.check(lib.sf_plan_set_wait_limit(s._plan, 0, 0), "sf_plan_set_wait_limit")
    s.reset()
    s.run_steps(10)
    for f, v in saved.items():
        np.testing.assert_array_equal(getattr(s, f), v, err_msg=f)
    s.run_steps(10)
    ref.run_steps(10)
    for f in FIELDS:
        np.testing.assert_array_equal(getattr(s, f), getattr(ref, f), err_msg=f)


@pytest.mark.parametrize("boundary", ["abc", "radiation", "pml"])
@pytest.mark.parametrize("shape", [(33, 29, 31), (61, 50, 66), (112, 96, 120), (66, 130, 97)])
def test_what_acts_between_the_steps_against_single_steps(shape, boundary):
    """Plane boundaries, membranes that overlap a point and a plane source,
    omnidirectional and directional microphones on and off block edges: the
    same run with the per-step kernels gives the same fields, traces and
    waveforms, over two calls and after a reset."""
    r = 1e-3
    ext = [n * r for n in shape]

    def build():
        s = S.FDTDSolver(shape=shape, resolution=r, c=343.0, rho=1.2, courant=0.6)
        if boundary == "pml":
            s.add_boundary(S.PML(depth=4))
        elif boundary == "abc":
            s.add_boundary(S.ABCFirstOrder())
        else:
            s.add_boundary(S.PML(depth=4, axis="y"))
            s.add_boundary(S.ABCFirstOrder(axis="z"))
            s.add_boundary(S.RadiationImpedance("x", "low", reflection_coeff=0.3))
            s.add_boundary(S.RadiationImpedance("x", "high", pipe_radius=0.01))
        s.add_source(S.CircularMembraneSource(
            center=(ext[0] / 2, ext[1] / 2, 10.5 * r), normal_axis="z", radius=9 * r, mode=(1, 1),
            waveform=S.GaussianPulse(position=(0, 0, 0), frequency=20000.0)))
        s.add_source(S.GaussianPulse(position=(shape[0] // 2, shape[1] // 2, 10), frequency=15000.0))
        s.add_source(S.RectangularMembraneSource(
            center=(12.5 * r, ext[1] / 2, ext[2] / 2), normal_axis="x", size=(15 * r, 12 * r),
            waveform=S.GaussianPulse(position=(0, 0, 0), frequency=18000.0)))
        s.add_source(S.GaussianPulse(position={"axis": 1, "index": 7}, frequency=9000.0,
                                     amplitude=0.1, source_type="plane"))
        s.add_probe("a", (0, 0, 0))
        s.add_probe("b", tuple(n - 1 for n in shape))
        s.add_microphone(position=tuple(0.5 * e for e in ext), name="omni")
        s.add_microphone(position=tuple(0.31 * e for e in ext), name="card", pattern="cardioid",
                         direction=(1, 2, 0.5))
        s.add_microphone(position=(0.0002, 0.0007, ext[2] - 1.5 * r), name="edge", pattern="figure8",
                         direction=(0, 1, 0))
        return s

    a, b = build(), build()
    b.set_kernel("tile1_r2_w8")
    a._sync_tables()
    assert _native.load().sf_plan_resident(a._plan, 13, 1, a._stream())
    rng = np.random.default_rng(4)
    p0 = (rng.standard_normal(shape) * 1e-2).astype(np.float32)
    for again in (False, True):
        for s in (a, b):
            if again:
                s.reset()
            s.p = p0.copy()
            s.run_steps(13)
            s.run_steps(20)
        _check(a, b, (shape, boundary, again))
        for name in ("omni", "card", "edge"):
            np.testing.assert_array_equal(a.microphones[name].get_waveform(),
                                          b.microphones[name].get_waveform(), err_msg=name)


@pytest.mark.parametrize("scale", [1e-2, 1e-20, 1e-36, 1e36])
@pytest.mark.parametrize("courant", [0.6, 0.31])
def test_absorbing_planes_round_as_in_fp64(scale, courant):
    """The planes' FP64 operations in FP32 pairs, from magnitudes near both ends of
    the range (overflow included) and over zeros: the bits of the per-step kernel."""
    shape = (40, 37, 44)
    rng = np.random.default_rng(8)
    p0 = (rng.standard_normal(shape) * np.exp2(rng.integers(-20, 1, shape)) * scale).astype(np.float32)
    p0[rng.random(shape) < 0.3] = 0.0
    p0[:, :, 22:] *= rng.random() < 0.5
    out = []
    for kernel in (None, "tile1_r2_w8"):
        s = S.FDTDSolver(shape=shape, resolution=1e-3, c=343.0, rho=1.2, courant=courant)
        s.add_boundary(S.ABCFirstOrder())
        if kernel:
            s.set_kernel(kernel)
        else:
            assert _resident(s, 40)
        s.p = p0.copy()
        for n in (40, 9):
            s.run_steps(n)
        out.append(s)
    with np.errstate(all="ignore"):
        _check(*out, (scale, courant))
