"""The voxeliser with solids of many parts, of which a block looks only at those
that matter in it: every cell is sdf(cell centre) <= 0 of the whole program."""
import numpy as np
import pytest

import strata_fdtd_gb300 as S

pytestmark = pytest.mark.gpu

R = 1e-3


def _balls(n, seed, r=(2.0, 7.0), span=64):
    g = np.random.default_rng(seed)
    return [S.Sphere(center=tuple(g.uniform(0, span, 3) * R), radius=float(g.uniform(*r)) * R)
            for _ in range(n)]


def _boxes(n, seed):
    g = np.random.default_rng(seed)
    return [S.Box(center=tuple(g.uniform(4, 60, 3) * R), size=tuple(g.uniform(3, 22, 3) * R))
            for _ in range(n)]


def _resonators(n):
    out = []
    for q in range(n):
        x, y = 8 + 12 * (q % 5), 8 + 12 * (q // 5)
        out.append(S.Union(S.Cylinder(p1=(x * R, y * R, 30 * R), p2=(x * R, y * R, 50 * R), radius=1.5 * R),
                           S.Sphere(center=(x * R, y * R, 28 * R), radius=(3 + q % 3) * R)))
    return out


SHAPES = {
    "union": lambda: S.Union(*_balls(20, 1)),
    "more_than_the_markers": lambda: S.Union(*_balls(90, 2)),
    "outer_marked_inner_not": lambda: S.Difference(S.Union(*_boxes(40, 3)), *_resonators(25)),
    "resonator_array": lambda: S.Difference(
        S.Box(center=(32 * R, 32 * R, 30 * R), size=(60 * R, 58 * R, 40 * R)), *_resonators(20)),
    "intersection": lambda: S.Intersection(*[b for b in _balls(6, 4, (25.0, 40.0))]),
    "transformed_parts": lambda: S.Difference(
        S.Union(*[b.rotate_z(0.1 * q).translate((q * R, 0, -q * R)) for q, b in enumerate(_boxes(8, 5))])
        .rotate((1, 2, 3), 0.4),
        S.Union(*[b.scale(0.8).translate((3 * R, 2 * R, R)) for b in _balls(9, 6)]).scale(1.1),
        S.Intersection(*_balls(2, 7, (10.0, 20.0)))),
    "smooth_of_groups": lambda: S.SmoothUnion(S.Union(*_balls(5, 8)),
                                              S.Difference(S.Union(*_boxes(3, 9)), *_balls(3, 10)),
                                              radius=3 * R),
    "equal_parts": lambda: S.Union(*(_balls(3, 11) * 3), S.Union()),
    "nothing_but_itself_removed": lambda: S.Difference(*(_balls(1, 12, (9.0, 10.0)) * 2)),
}


@pytest.mark.parametrize("shape", [(64, 61, 70), (33, 70, 40), (1, 3, 130)])
@pytest.mark.parametrize("name", list(SHAPES))
def test_mask_equals_point_evaluation(name, shape):
    solid = SHAPES[name]()
    grid = S.UniformGrid(shape, R)
    pts = np.stack(np.meshgrid(grid.x_coords, grid.y_coords, grid.z_coords, indexing="ij"), -1)
    want = solid.contains(pts.reshape(-1, 3)).reshape(shape)
    assert np.array_equal(solid.voxelize(grid), want)
    assert np.array_equal(solid.voxelize_device(grid, invert=True).cpu().numpy().astype(bool), ~want)


@pytest.mark.parametrize("name", list(SHAPES))
def test_grid_of_many_super_blocks_equals_point_evaluation(name):
    """Thin, but with more super-blocks than are needed to look at those first."""
    solid = SHAPES[name]().translate((-30 * R, -29 * R, 0))
    grid = S.UniformGrid((17, 20, 16400), R / 256)
    pts = np.stack(np.meshgrid(grid.x_coords, grid.y_coords, grid.z_coords, indexing="ij"), -1)
    want = solid.contains(pts.reshape(-1, 3)).reshape(grid.shape)
    assert np.array_equal(solid.voxelize(grid), want)
