"""The tiled and the spread-cloud scoring kernels against the generic kernel
(which other tests pin to the oracle): the same fixed-point sums give the same
raw weights bit for bit, and the hit counts are equal -- at the edges of their
chunks, groups and regions, on maps whose bricks alias at the far edges, for
likelihoods too large for the default scale, and for batches with long items."""
import ctypes as C

import numpy as np
import pytest

from tsdf_localization_gb300 import Context, DeviceMap, FilterBatch, TSDFEvaluator, code_values
from tsdf_localization_gb300 import _native as N
from tsdf_localization_gb300 import synth

pytestmark = pytest.mark.gpu
LAYOUTS = {"compact": {"dense": True}, "brick": {}, "hash": {"hash_index": True}, "grid": {"grid": True}}


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def random_map(size, res: float, low, seed: int):
    """(coef, brick table, codes) of a map of `size` metres with random bricks
    and codes; coefficients as the CudaSubVoxelMap constructor forms them."""
    rng = np.random.default_rng(seed)
    c = N.MapCoef()
    f = np.float32
    lo, hi = np.array(low, f), np.array(low, f) + np.array(size, f)
    dim = [int(np.ceil(f(abs(h - l)) / f(res))) for l, h in zip(lo, hi)]
    up = [int(np.ceil(f(abs(h - l)))) for l, h in zip(lo, hi)]
    c.dim_x, c.dim_y, c.dim_z = dim
    c.min_x, c.min_y, c.min_z = (float(v) for v in lo)
    c.max_x, c.max_y, c.max_z = (float(v) for v in hi)
    c.resolution, c.init_value = res, 0.0
    c.up_dim_x, c.up_dim_y, c.up_dim_z = up
    c.up_dim_2 = up[0] * up[1]
    c.sub_dim = int(np.ceil(f(1.0) / f(res)))
    c.sub_dim_2 = c.sub_dim ** 2
    c.grid_occ_size = up[0] * up[1] * up[2]
    have = rng.random(c.grid_occ_size) < 0.8
    occ = np.where(have, (np.cumsum(have) - 1) * c.sub_dim ** 3, -1).astype(np.int32)
    c.data_size = int(have.sum()) * c.sub_dim ** 3
    return c, occ, rng.integers(0, 601, c.data_size, dtype=np.uint16)


def cloud(spread: bool, P: int, size, low, rng):
    p = np.zeros((P, 7), np.float32)
    span = np.array(size) if spread else np.array([1.0, 1.0, 1.0])
    base = np.array(low) if spread else np.array(low) + np.array(size) / 2
    p[:, :3] = base + rng.random((P, 3)) * span
    p[:, 2] = low[2] + 0.3 + rng.random(P)
    p[:, 3:5] = rng.normal(0, 0.03, (P, 2))
    p[:, 5] = rng.uniform(-np.pi, np.pi, P)
    if spread:   # the extent that makes a cloud spread, whatever the draws
        p[0, :2], p[-1, :2] = base[:2], base[:2] + span[:2]
    return p


def scan(n: int, rng):
    """Points up to 8 m away, a few far outside the map, one not finite."""
    q = rng.normal(0, 4, (n, 3)).astype(np.float32)
    q[:, 2] *= 0.4
    if n > 20:
        q[7] = (300.0, -5.0, 1.0)
        q[11] = (2.0, np.nan, 0.0)
        q[13] = (-1e9, 3.0, 0.0)
    return q


def same(ctx, dmap, parts, pts, tf=synth.IDENTITY_TF):
    fast = TSDFEvaluator(dmap).evaluate_debug(parts.copy(), pts, tf)
    ref = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, tf)
    assert np.array_equal(fast["hits"], ref["hits"])
    assert np.array_equal(fast["raw"], ref["raw"])
    assert ref["hits"].any() or parts.shape[0] * pts.shape[0] < 100   # a lookup or two may all miss


SIZES = {False: ((2, 1), (15, 63), (16, 64), (17, 65), (33, 127), (64, 128), (65, 129), (250, 1024), (251, 1025),
                 (20_000, 257), (40, 17_000)),
         # at least kOrderFrom lookups: the spread kernel
         True: ((400_009, 126), (400_000, 128), (395_001, 129), (800_000, 64), (800_001, 65), (16_401, 3203),
                (16_384, 3072), (3001, 17_000))}


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("low", [(0.0, 0.0, 0.0), (-3.25, 1.5, -0.5)])
@pytest.mark.parametrize("spread", [False, True])
def test_chunk_group_and_region_edges(ctx, layout, low, spread):
    size = (21.3, 17.6, 5.2)
    rng = np.random.default_rng(3)
    coef, occ, codes = random_map(size, 0.1, low, 1)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, **LAYOUTS[layout])
    assert dmap.info()["fast_index"]
    for P, n in SIZES[spread]:
        assert not spread or P * n >= 3 << 24
        same(ctx, dmap, cloud(spread, P, size, low, rng), scan(n, rng))


@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_bricks_that_alias_at_the_far_edge(ctx, layout):
    """Sizes of whole metres at 0.064 m: the last brick coordinate that passes the
    coarse check equals the table's size, so brick indices reach past its rows."""
    size = (21.0, 17.0, 4.0)
    rng = np.random.default_rng(4)
    coef, occ, codes = random_map(size, 0.064, (0, 0, 0), 2)
    assert int(np.float32(21.0) / np.float32(0.064)) < coef.dim_x and coef.up_dim_x == 21
    dmap = DeviceMap(ctx, coef, occ, codes=codes, **LAYOUTS[layout])
    for spread, P in ((False, 500), (True, 73_000)):
        parts = cloud(spread, P, size, (0, 0, 0), rng)
        parts[1:250, :3] = np.array(size) - rng.random((249, 3)) * 0.2
        same(ctx, dmap, parts, scan(700, rng))


@pytest.mark.parametrize("sigma", [0.02, 0.05, 0.1])
def test_likelihood_scale(ctx, sigma):
    """Peak likelihoods of 7,937, 508 and 63.5: the sums against FP64 sums of the
    slots' values, within the fixed point's resolution and one float rounding."""
    size = (12.5, 11.5, 4.5)
    rng = np.random.default_rng(5)
    coef, occ, codes = random_map(size, 0.1, (0, 0, 0), 3)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, sigma=sigma, dense=True)
    for n in (100, 3000):
        parts, pts = cloud(False, 64, size, (0, 0, 0), rng), scan(n, rng)
        d = TSDFEvaluator(dmap).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF, voxel_index=True)
        same(ctx, dmap, parts, pts)
        values = np.append(code_values(sigma), [0.0]).astype(np.float64)   # 601: a miss
        sums = values[np.minimum(d["voxel_index"] & 0xFFFF, 601)].sum(1)
        inside = (pts.astype(np.float64) ** 2).sum(1) < 1e4
        want = np.float32(0.9) * sums + inside.sum() * np.float64(np.float32(0.1) * np.float32(0.01))
        # n values rounded to at most 2^-34 of a unit each, one float rounding
        assert np.all(np.abs(d["raw"] - want) <= 0.9 * n * 2.0 ** -35 + 2.0 ** -23 * want)


def test_batch_with_long_items(ctx):
    """Items of 4,096 points unpack their sums several times."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(6)
    size = (21.3, 17.6, 5.2)
    coef, occ, codes = random_map(size, 0.1, (0, 0, 0), 4)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, dense=True)
    filters, keep = [], []
    for P, n in ((50, 5000), (7, 9001)):
        parts, pts = cloud(False, P, size, (0, 0, 0), rng), scan(n, rng)
        d = [torch.from_numpy(parts.copy()).cuda(), torch.from_numpy(pts).cuda(), torch.zeros(6, device="cuda")]
        keep.append((parts, pts, d))
        filters.append({"map": dmap, "P": P, "N": n, "tf": synth.IDENTITY_TF, "particles": d[0].data_ptr(),
                        "points": d[1].data_ptr(), "pose_out": d[2].data_ptr()})
    torch.cuda.synchronize()
    b = FilterBatch(ctx, filters)
    for tiles in ((4096, 2), (1024, 4), (192, 1)):
        b.set_tiles(*tiles)
        b.run()
        ctx.sync()
        for i, (parts, pts, d) in enumerate(keep):
            want = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
            assert np.array_equal(b.hits(i, parts.shape[0]), want["hits"])
            w = (want["raw"] / np.float32(want["weight_sum"])).astype(np.float32)
            assert np.array_equal(d[0].cpu().numpy()[:, 6], w)
    b.close()
