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
