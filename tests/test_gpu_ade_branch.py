"""ADE steps captured into a graph run the material boxes beside the plain
cells; single steps run the two in turn."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import cases as C  # noqa: E402
import strata_fdtd_gb300 as S  # noqa: E402
from test_gpu_parity import API  # noqa: E402


@pytest.mark.parametrize("name", ["split_boxes_geom", "lorentz_mixed_geom", "nu_mixed_geom",
                                  "materialized_sdf"])
def test_captured_ade_steps_equal_single_steps(name):
    """150 steps from graphs, of a grid wide enough for warp tiles beside the
    boxes, and the same 150 one by one: equal bits in fields, J and traces."""
    out = []
    for single in (False, True):
        s = C.build_case(API, C.ADE_CASES[name])
        if single:
            for _ in range(150):
                s.step()
        else:
            s.run_steps(150)
        fields = [np.asarray(f).copy() for f in (s.p, s.vx, s.vy, s.vz)]
        j = []
        if s._ade_debye:
            j.append(np.array(s._ade_J_debye))
        if s._ade_lorentz:
            j += [np.array(s._ade_J_lorentz), np.array(s._ade_J_lorentz_prev)]
        out.append((fields + j, s.get_probe_data()))
    (a, ta), (b, tb) = out
    assert len(a) > 4 and len(a) == len(b)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    assert list(ta) == list(tb)
    for k in ta:
        np.testing.assert_array_equal(ta[k], tb[k])


MODULUS_ONLY = dict(
    shape=(40, 45, 140), res=1e-3, courant=0.5, pml=dict(depth=5),
    materials=[dict(id=2, name="m2", rho=1.3, c=330.0, poles=[("debye", "modulus", 0.3, 4e-4)],
                    box=((19, 31), (13, 27), (33, 47))),
               dict(id=5, name="m5", rho=1.1, c=355.0,
                    poles=[("lorentz", "modulus", 0.15, 2 * np.pi * 9000.0, 4000.0)],
                    box=((30, 37), (20, 31), (45, 52)))],
    sources=[("point", (20, 22, 38), 15000.0, 1.0), ("point", (10, 30, 60), 11000.0, 0.6)],
    probes=[("mid", (25, 20, 40)), ("far", (30, 35, 20)), ("wide", (20, 22, 120))],
    steps=100, store_fields=False)


def test_captured_steps_of_modulus_poles_alone_equal_single_steps(monkeypatch):
    """Without a density pass the per-cell kernel is the first launch of the branch."""
    monkeypatch.setitem(C.ADE_CASES, "modulus_only", MODULUS_ONLY)
    test_captured_ade_steps_equal_single_steps("modulus_only")
