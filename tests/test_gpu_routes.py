"""Routes of the automatic kernel choice that the tests of each kernel leave out:
what acts between the steps on the chip with walls and on stretched grids, a call
captured by the caller, the two-step windows without walls and at full size."""
import numpy as np
import pytest

import cases as C
from conftest import sha256

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402
from strata_fdtd_gb300 import _native  # noqa: E402
from oracle import oracle as O  # noqa: E402

from test_gpu_parity import API  # noqa: E402
from test_gpu_pipe import _case, _check  # noqa: E402
from test_gpu_tb import _case as tb_case  # noqa: E402

WINDOWS = [c for c in S.solver.kernel_configs() if c.startswith("tb2q")]


# the kinds of 1, 2, 4 and 8 planes per thread
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("shape", [(33, 29, 31), (58, 50, 66), (80, 76, 84), (100, 96, 92), (110, 104, 108)])
def test_what_acts_between_the_steps(shape, walls, stretched):
    """Absorbing planes, a membrane, a point source and microphones (one a cardioid) with
    walls and on stretched grids, against the per-step kernels."""
    r = 1e-3
    rng = np.random.default_rng(sum(shape))
    coords = [np.cumsum(rng.uniform(0.8, 1.25, n)) * r for n in shape]
    mask = np.ones(shape, bool)
    mask[shape[0] // 3:shape[0] // 3 + 7, 5:20, 6:25] = False
    mask[-4:, :9, -5:] = False

    def build():
        if stretched:
            s = S.FDTDSolver(grid=S.NonuniformGrid(*coords), c=343.0, rho=1.2, courant=0.6)
        else:
            s = S.FDTDSolver(shape=shape, resolution=r, c=343.0, rho=1.2, courant=0.6)
        s.add_boundary(S.PML(depth=4, axis="y"))
        s.add_boundary(S.ABCFirstOrder(axis="z"))
        s.add_boundary(S.RadiationImpedance("x", "low", reflection_coeff=0.3))
        if walls:
            s.set_geometry(mask.copy())
        ext = [float(c[-1]) for c in coords] if stretched else [n * r for n in shape]
        s.add_source(S.CircularMembraneSource(
            center=(ext[0] / 2, ext[1] / 2, 3.5 * r), normal_axis="z", radius=6 * r, mode=(0, 1),
            waveform=S.GaussianPulse(position=(0, 0, 0), frequency=20000.0)))
        s.add_source(S.GaussianPulse(position=(shape[0] // 2, shape[1] // 2, 3), frequency=15000.0))
        s.add_probe("a", tuple(n // 2 for n in shape))
        s.add_microphone(position=tuple(0.5 * e for e in ext), name="omni")
        s.add_microphone(position=tuple(0.61 * e for e in ext), name="card", pattern="cardioid",
                         direction=(1, 2, 0.5))
        return s

    a, b = build(), build()
    b.set_kernel("tile1_r2_w8")
    a._sync_tables()
    assert _native.load().sf_plan_resident(a._plan, 11, 1, a._stream())
    p0 = (rng.standard_normal(shape) * 1e-2).astype(np.float32) * (mask if walls else 1)
    for s in (a, b):
        s.p = p0.copy()
        s.run_steps(11)
        s.run_steps(16)
    _check(a, b, (shape, walls, stretched))
    for name in ("omni", "card"):
        np.testing.assert_array_equal(a.microphones[name].get_waveform(),
                                      b.microphones[name].get_waveform(), err_msg=name)


@pytest.mark.parametrize("shape", [(40, 41, 44), (70, 45, 76), (131, 204, 168)])
def test_steps_captured_by_the_caller(shape):
    """A graph of 20 steps captured by the caller (which takes the kernels of single or
    paired steps) and replayed three times equals 60 steps."""
    case = _case(shape, 0)
    s, ref = (C.build_case(API, case) for _ in range(2))
    for x in (s, ref):
        x.run_steps(2)
    n = len(s._probe_order)
    src = s.source_table(20)
    trace = torch.zeros((20, n), dtype=torch.float32, device="cuda")
    lib, stream = _native.load(), torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        rc = lib.sf_plan_step(s._plan, 20, src.data_ptr(), trace.data_ptr(), stream.cuda_stream)
    assert rc == 0
    names = list(s._probe_order)
    samples = [s.get_probe_data()[q] for q in names]
    for rep in range(3):
        src.copy_(s.source_table(20))
        g.replay()
        samples = [np.concatenate([v, trace[:, q].cpu().numpy()]) for q, v in enumerate(samples)]
        for _ in range(20):
            s._time += s.dt
    s._mark_device_newer()
    ref.run_steps(60)
    for f in ("p", "vx", "vy", "vz"):
        np.testing.assert_array_equal(getattr(s, f), getattr(ref, f), err_msg=f)
    for name, v in zip(names, samples):
        np.testing.assert_array_equal(v, ref.get_probe_data()[name], err_msg=name)


@pytest.mark.parametrize("config", WINDOWS)
@pytest.mark.parametrize("shape", [(40, 48, 96), (31, 70, 168), (17, 33, 40)])
def test_windows_without_walls(config, shape):
    case = tb_case(shape, 50, geometry=False)
    ref = C.build_case(O.make_api(), case)
    ref.run_steps(50)
    s = C.build_case(API, case)
    s.set_kernel(config, 0)
    s.run_steps(50)
    _check(s, ref, (config, shape))


def test_windows_at_full_size():
    """The 400^3 enclosure from a random state: 12 steps of each window configuration
    equal 12 single steps of the warp-tile kernel."""
    solid = C.c2_solid(API)
    init = None
    sums = []
    for kernel in ["tile_r1_w4_m6"] + WINDOWS:
        s = S.FDTDSolver(shape=(400, 400, 400), resolution=1e-3, c=343.0, rho=1.204, courant=0.5)
        s.add_boundary(S.PML(depth=16))
        s.set_geometry_sdf(solid)
        s.add_source(S.GaussianPulse(position=(200, 200, 200), frequency=2000.0))
        for q, pos in enumerate(((200, 200, 230), (0, 0, 0), (399, 399, 399), (201, 7, 79))):
            s.add_probe(f"p{q}", pos)
        if init is None:
            init = np.random.default_rng(11).standard_normal((400, 400, 400), dtype=np.float32)
            init *= np.float32(1e-3)
            init[~s.geometry] = 0.0
        s.p = init.copy()
        s.set_kernel(kernel)
        s.run_steps(12)
        sums.append([sha256(getattr(s, f)) for f in ("p", "vx", "vy", "vz")]
                    + [v.tolist() for v in s.get_probe_data().values()])
        del s
    assert all(x == sums[0] for x in sums[1:])
