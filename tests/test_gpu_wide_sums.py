"""Small sigma: likelihoods too large for the packed sums, so the wide form of the tiled,
spread, subsampling and batch kernels.  Raw weights and hits equal the generic
kernel's bit for bit, and the raw weights are as close to FP64 sums as the largest
scale that 62 bits allow: a range term of 0 and a map of distances far out in the
tail leave particles whose whole weight is a few units of that scale."""
import numpy as np
import pytest

from tsdf_localization_gb300 import Context, DeviceMap, FilterBatch, TSDFEvaluator, code_values
from tsdf_localization_gb300 import synth

from test_gpu_scoring_kernels import LAYOUTS, cloud, random_map, scan

pytestmark = pytest.mark.gpu
SIZE = (21.3, 17.6, 5.2)


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def scale_shift(top: float, n: int) -> int:
    return min(40, 62 - int(np.ceil(np.log2(top * (n + 1.0)))))


def model(**kw):
    return dict(a_hit=0.9, a_range=0.0, a_max=0.0, **kw)


@pytest.mark.parametrize("sigma,codes_of", [(0.005, (22, 25)), (0.01, (40, 46)), (0.02, (80, 92)), (0.005, (0, 601)),
                                            (0.04, (0, 601)), (0.1, (0, 601))])
@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_sums_keep_their_scale(ctx, layout, sigma, codes_of):
    rng = np.random.default_rng(1)
    coef, occ, codes = random_map(SIZE, 0.1, (0, 0, 0), 1)
    codes = rng.integers(*codes_of, codes.shape[0], dtype=np.uint16)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, sigma=sigma, **LAYOUTS[layout])
    values = np.append(code_values(sigma), [0.0]).astype(np.float64)
    for n in (1, 33, 100, 1000, 3001, 5000):
        parts, pts = cloud(False, 100, SIZE, (0, 0, 0), rng), scan(n, rng)
        fast = TSDFEvaluator(dmap, **model()).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        ref = TSDFEvaluator(dmap, generic=True, **model()).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        assert np.array_equal(fast["hits"], ref["hits"]) and np.array_equal(fast["raw"], ref["raw"])
        d = TSDFEvaluator(dmap, **model()).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF, voxel_index=True)
        assert np.array_equal(d["hits"], ref["hits"]) and np.array_equal(d["raw"], ref["raw"])
        want = np.float64(np.float32(0.9)) * values[np.minimum(d["voxel_index"] & 0xFFFF, 601)].sum(1)
        # n values rounded to half a unit of the scale each, one rounding to float
        unit = 2.0 ** -scale_shift(float(values.max()), n)
        assert np.all(np.abs(fast["raw"] - want) <= 0.9 * n * unit / 2 + 2.0 ** -23 * want)


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("low", [(0.0, 0.0, 0.0), (-3.25, 1.5, -0.5)])
def test_spread_clouds(ctx, layout, low):
    rng = np.random.default_rng(2)
    coef, occ, codes = random_map(SIZE, 0.1, low, 2)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, sigma=0.005, **LAYOUTS[layout])
    for P, n in ((400_009, 126), (395_001, 129), (16_401, 3203)):
        parts, pts = cloud(True, P, SIZE, low, rng), scan(n, rng)
        fast = TSDFEvaluator(dmap, **model()).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        ref = TSDFEvaluator(dmap, generic=True, **model()).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        assert np.array_equal(fast["hits"], ref["hits"]) and np.array_equal(fast["raw"], ref["raw"])


@pytest.mark.parametrize("layout", ["compact", "brick"])
@pytest.mark.parametrize("res", [0.1, 0.064])   # one- and two-term sub-voxel multipliers
def test_subsampled_and_batched(ctx, layout, res):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    coef, occ, codes = random_map(SIZE, res, (0, 0, 0), 3)
    dmaps = [DeviceMap(ctx, coef, occ, codes=codes, sigma=s, **LAYOUTS[layout]) for s in (0.005, 0.1, 0.03)]
    filters, keep = [], []
    for i, (P, n) in enumerate(((50, 100), (7, 3001), (333, 700), (64, 65), (5, 14_001), (90, 64), (40_000, 400))):
        dmap = dmaps[i % 3]
        parts, pts = cloud(False, P, SIZE, (0, 0, 0), rng), scan(n, rng)
        want = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        # every point kept: the subsampling kernel gives the whole scan's sums
        _, raw, hits = TSDFEvaluator(dmap).evaluate_subsampled(parts.copy(), pts, synth.IDENTITY_TF, n, 5, debug=True)
        assert np.array_equal(raw, want["raw"]) and np.array_equal(hits, want["hits"])
        d = [torch.from_numpy(parts.copy()).cuda(), torch.from_numpy(pts).cuda(), torch.zeros(6, device="cuda")]
        keep.append((parts, d, want))
        filters.append({"map": dmap, "P": P, "N": n, "tf": synth.IDENTITY_TF, "particles": d[0].data_ptr(),
                        "points": d[1].data_ptr(), "pose_out": d[2].data_ptr()})
    torch.cuda.synchronize()
    b = FilterBatch(ctx, filters)
    for tiles in ((4096, 2), (1024, 4), (192, 1)):
        b.set_tiles(*tiles)
        for parts, d, _ in keep:
            d[0].copy_(torch.from_numpy(parts))
        torch.cuda.synchronize()
        b.run()
        ctx.sync()
        for i, (parts, d, want) in enumerate(keep):
            assert np.array_equal(b.hits(i, parts.shape[0]), want["hits"])
            w = (want["raw"] / np.float32(want["weight_sum"])).astype(np.float32)
            assert np.array_equal(d[0].cpu().numpy()[:, 6], w)
    b.close()
