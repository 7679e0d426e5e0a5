"""The block-wise voxeliser against the point evaluator: every mask cell is
sdf(cell centre) <= 0 of the FP64 program, whatever decided it (a 4 x 4 x 4
block's interval, a cell's interval, or the FP64 evaluation itself)."""
import numpy as np
import pytest

import strata_fdtd_gb300 as S

pytestmark = pytest.mark.gpu

R = 1e-3


def _box(c=(12, 12, 12), s=(14, 10, 16)):
    return S.Box(center=tuple(v * R for v in c), size=tuple(v * R for v in s))


def _ball(c=(12.5, 12.5, 12.5), r=8.0):
    return S.Sphere(center=tuple(v * R for v in c), radius=r * R)


def _pipe(p=(4, 12, 12), q=(21, 12, 12), r=5.0):
    return S.Cylinder(p1=tuple(v * R for v in p), p2=tuple(v * R for v in q), radius=r * R)


def _horn(profile):
    return S.Horn(throat_position=(12 * R, 12 * R, 3 * R), mouth_position=(12 * R, 12 * R, 21 * R),
                  throat_radius=3 * R, mouth_radius=9 * R, profile=profile)


SHAPES = {
    "box": _box,
    "box_faces_on_centres": lambda: _box((12.5, 12.5, 12.5), (12, 10, 16)),
    "sphere": _ball,
    "sphere_through_centres": lambda: _ball((12.5, 12.5, 12.5), 5.0),
    "cylinder_axis": _pipe,
    "cylinder_oblique": lambda: _pipe((3, 5, 4), (20, 18, 22), 4.0),
    "cone": lambda: S.Cone(p1=(12 * R, 12 * R, 3 * R), p2=(13 * R, 10 * R, 21 * R), r1=8 * R,
                           r2=2 * R),
    "horn_conical": lambda: _horn("conical"),
    "horn_exponential": lambda: _horn("exponential"),
    "horn_hyperbolic": lambda: _horn("hyperbolic"),
    "horn_tractrix": lambda: _horn("tractrix"),
    "csg": lambda: S.Union(S.Difference(_box(), _ball()), S.Intersection(_pipe(), _ball(r=6.0))),
    "empty_union": lambda: S.Union(),
    "smooth": lambda: S.SmoothUnion(_box(), _pipe(), radius=2 * R),
    "smooth_intersection": lambda: S.SmoothIntersection(_box(), _ball(), radius=2 * R),
    "smooth_difference": lambda: S.SmoothDifference(_box(), _ball(r=5.0), radius=2 * R),
    "transforms": lambda: S.Difference(_box().rotate_z(0.3).translate((1 * R, -2 * R, 0)),
                                       _ball().scale(0.7).rotate((1, 2, 3), 0.5)),
    "far_translation": lambda: _ball().translate((1e6, 0, 0)).translate((-1e6, 0, 0)),
    "spiral": lambda: S.SpiralHorn(center=(12 * R, 12 * R), throat_radius=1 * R, mouth_radius=3 * R,
                                   inner_spiral_radius=3 * R, outer_spiral_radius=9 * R, turns=1.5,
                                   height=15 * R),
    "helix": lambda: S.HelicalTube(center=(12 * R, 12 * R, 4 * R), helix_radius=7 * R,
                                   tube_radius_start=1 * R, tube_radius_end=2.5 * R, pitch=6 * R,
                                   turns=2),
}


@pytest.mark.parametrize("shape", [(25, 24, 23), (24, 25, 28), (1, 3, 130)])
@pytest.mark.parametrize("name", list(SHAPES))
def test_mask_equals_point_evaluation(name, shape):
    solid = SHAPES[name]()
    grid = S.UniformGrid(shape, R)
    pts = np.stack(np.meshgrid(grid.x_coords, grid.y_coords, grid.z_coords, indexing="ij"), -1)
    want = solid.contains(pts.reshape(-1, 3)).reshape(shape)
    assert np.array_equal(solid.voxelize(grid), want)
    assert np.array_equal(solid.voxelize_device(grid, invert=True).cpu().numpy().astype(bool), ~want)


@pytest.mark.parametrize("name", ["csg", "horn_tractrix", "transforms"])
def test_stretched_grid_equals_point_evaluation(name):
    solid = SHAPES[name]()
    rng = np.random.default_rng(3)
    grid = S.NonuniformGrid(*(np.cumsum(rng.uniform(0.4, 1.6, n)) * R for n in (27, 22, 31)))
    pts = np.stack(np.meshgrid(grid.x_coords, grid.y_coords, grid.z_coords, indexing="ij"), -1)
    want = solid.contains(pts.reshape(-1, 3)).reshape(grid.shape)
    assert np.array_equal(solid.voxelize(grid), want)


@pytest.mark.parametrize("stretched", [False, True])
def test_slabs_of_a_large_grid(stretched):
    """270 million cells of a thin grid are done in two slabs of planes: cells of the
    planes around their border, and cells drawn from the whole grid."""
    shape = (450, 5, 120001)
    rng = np.random.default_rng(7)
    if stretched:
        coords = [np.cumsum(rng.uniform(0.7, 1.3, n)) * R for n in shape]
        grid = S.NonuniformGrid(*coords)
    else:
        coords = [np.arange(n) * R + R / 2 for n in shape]
        grid = S.UniformGrid(shape, R)
    solid = S.Difference(
        S.Union(S.Cylinder(p1=(0.2, 0.002, 0.0), p2=(0.25, 0.003, 121.0), radius=0.1),
                S.Sphere(center=(0.24, 0.002, 60.0), radius=0.21)),
        S.Sphere(center=(0.23, 0.0025, 30.0), radius=0.05))
    mask = solid.voxelize(grid)
    cells = [rng.integers(0, n, 1_000_000) for n in shape]
    border = [rng.integers(236, 244, 300_000), rng.integers(0, 5, 300_000),
              np.concatenate([rng.integers(0, 120001, 100_000), rng.integers(59700, 60300, 100_000),
                              rng.integers(29900, 30100, 100_000)])]
    for i, j, k in (cells, border):
        points = np.stack([coords[0][i], coords[1][j], coords[2][k]], axis=1)
        np.testing.assert_array_equal(mask[i, j, k], solid.contains(points))
        assert 0.02 < mask[i, j, k].mean() < 0.98
