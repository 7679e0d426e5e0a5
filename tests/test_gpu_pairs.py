"""Pairs of steps by the automatic kernel choice: the same bits as single steps of
the warp-tile kernel, in calls of every remainder, graphs and a caller's capture."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402

FIELDS = ("p", "vx", "vy", "vz")


def _build(shape, walls, plane_axis):
    s = S.FDTDSolver(shape=shape, resolution=1e-3, c=343.0, rho=1.2, courant=0.55)
    s.add_boundary(S.PML(depth=6))
    if walls:
        m = np.ones(shape, bool)
        m[20:41, 11:60, :70] = False
        m[:, 80:84, 55:58] = False
        m[-9:, -3:, -5:] = False
        s.set_geometry(m)
    s.add_source(S.GaussianPulse(position=(70, 12, 56), frequency=9000.0))
    s.add_source(S.GaussianPulse(position=(71, 13, 55), frequency=7000.0))
    s.add_source(S.GaussianPulse(position={"axis": plane_axis, "index": 9}, frequency=5000.0,
                                 amplitude=0.1, source_type="plane"))
    for q, pos in enumerate(((0, 0, 0), tuple(n - 1 for n in shape), (70, 12, 56), (66, 23, 111))):
        s.add_probe("p%d" % q, pos)
    return s


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("shape,plane_axis", [((210, 132, 224), 0), ((210, 132, 223), 0),
                                              ((131, 204, 168), 0), ((131, 204, 168), 2)])
def test_automatic_choice_equals_single_steps(shape, plane_axis, walls):
    """2.5 to 6.2 million cells (too many to stay on chip), windows that end with the
    grid and short of it, odd nz on its padded twin, sources and probes on window
    edges, a plane source of either route; calls of 1 to 103 steps."""
    rng = np.random.default_rng(sum(shape))
    init = {f: (rng.standard_normal(shape) * 1e-2).astype(np.float32) for f in FIELDS}
    a, b = _build(shape, walls, plane_axis), _build(shape, walls, plane_axis)
    b.set_kernel("tile1_r4_w4")
    for s in (a, b):
        for f in FIELDS:
            v = init[f].copy()
            if f == "p":
                v[~s.geometry] = 0.0
            if f == "vz":
                v[:, :, -1] = 0.0
            setattr(s, f, v)
        for n in (1, 2, 3, 5, 8, 103, 50):
            s.run_steps(n)
    for f in FIELDS:
        np.testing.assert_array_equal(getattr(a, f), getattr(b, f), err_msg=f)
    ta, tb = a.get_probe_data(), b.get_probe_data()
    for k in tb:
        np.testing.assert_array_equal(ta[k], tb[k], err_msg=k)


def test_the_tuner_leaves_windows_out_with_a_plane_source_across_their_planes():
    a, b = _build((131, 204, 168), True, 2), _build((131, 204, 168), True, 0)
    names = [c for c in S.solver.kernel_configs() if c.startswith("tb2q")]
    assert not set(names) & set(a.autotune(launches=2))
    assert set(names) <= set(b.autotune(launches=2))
