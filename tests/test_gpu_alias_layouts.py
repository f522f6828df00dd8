"""Maps whose last brick coordinate that passes the coarse check lies past the brick
table (sizes of whole metres at a resolution that does not divide them): they get the
layout that was asked for -- the grid, and the bitmap up to its largest size -- and
score as the generic kernel does, below the floor, above the top and past the sides."""
import numpy as np
import pytest

from tsdf_localization_gb300 import Context, DeviceMap, TSDFEvaluator, synth

from test_gpu_scoring_kernels import cloud, random_map, scan

pytestmark = pytest.mark.gpu
GRID, BITMAP, HASH = 3, 1, 2


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def aliases(coef, axis: str) -> bool:
    up, dim = getattr(coef, "up_dim_" + axis), getattr(coef, "dim_" + axis)
    return int(np.float32(up) / np.float32(coef.resolution)) < dim


def check(ctx, dmap, size, rng, clouds):
    for spread, P, n in clouds:
        parts = cloud(spread, P, size, (0, 0, 0), rng)
        k = min(P - 2, 400)
        # at the far sides, below the floor and about the top
        parts[1:k, :3] = np.array(size) - rng.random((k - 1, 3)) * (0.4, 0.4, 0.0)
        parts[1:k:3, 2] = -rng.random(parts[1:k:3].shape[0])
        parts[2:k:3, 2] += rng.uniform(-1, 1, parts[2:k:3].shape[0])
        pts = scan(n, rng)
        pts[::2] *= np.float32(0.05)
        fast = TSDFEvaluator(dmap).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        ref = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        assert np.array_equal(fast["hits"], ref["hits"]) and np.array_equal(fast["raw"], ref["raw"])
        assert ref["hits"].any()


CLOUDS = ((False, 500, 1500), (True, 73_000, 700))


@pytest.mark.parametrize("size,res", [((21.3, 17.6, 4.0), 0.064), ((21.0, 17.0, 4.0), 0.064), ((21.0, 17.6, 4.2), 0.064),
                                      ((21.3, 17.0, 5.0), 0.3), ((21.3, 17.6, 4.2), 0.064)])
def test_grid_layout(ctx, size, res):
    rng = np.random.default_rng(1)
    coef, occ, codes = random_map(size, res, (0, 0, 0), 1)
    for axis, s in zip("xyz", size):
        assert aliases(coef, axis) == (s == int(s))
    dmap = DeviceMap(ctx, coef, occ, codes=codes, grid=True)
    assert dmap.info()["dense"] == GRID
    check(ctx, dmap, size, rng, CLOUDS)


@pytest.mark.parametrize("size,layout,table", [((100.0, 100.0, 52.0), BITMAP, 1 << 17), ((70.0, 71.0, 52.0), BITMAP, 1 << 16),
                                               ((100.0, 100.0, 53.0), HASH, 0), ((30.0, 31.0, 9.0), BITMAP, 1 << 12)])
def test_bitmap_up_to_its_largest_size(ctx, size, layout, table):
    """520,000 bricks of at most 524,288; 258,440 of the 262,144 of half the table."""
    rng = np.random.default_rng(2)
    coef, occ, codes = random_map(size, 0.3, (0, 0, 0), 2)
    assert aliases(coef, "z")
    plain = DeviceMap(ctx, coef, occ, codes=codes)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, dense=True)
    assert dmap.info()["dense"] == layout
    if table:
        assert dmap.info()["device_bytes"] - plain.info()["device_bytes"] == table
    check(ctx, dmap, size, rng, CLOUDS)
