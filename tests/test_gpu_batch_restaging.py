"""A block of the batch's scoring launch goes from segment to segment: the points (and
the bitmap) of the next one are copied over the place where the last one's deferred
lookups stood.  Segments of growing and shrinking scans on maps with and without a
bitmap, with many lookups that are deferred (coordinates that are not finite), few
items each, so that every block takes many segments."""
import numpy as np
import pytest

from tsdf_localization_gb300 import Context, DeviceMap, FilterBatch, TSDFEvaluator, synth

from test_gpu_scoring_kernels import cloud, random_map

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dense", [False, True])
def test_segments_over_each_others_rings(dense, captured):
    ctx = Context(0)
    rng = np.random.default_rng(12)
    size = (30.0, 25.0, 5.0)
    coef, occ, codes = random_map(size, 0.25, (0, 0, 0), 8)
    dmap = DeviceMap(ctx, coef, occ, codes=codes, dense=dense)
    filters, keep = [], []
    for i in range(48):
        P, n = 3 + i % 5, (64, 9000, 1025, 4097, 200, 6000)[i % 6] + 7 * i
        parts = cloud(False, P, size, (0, 0, 0), rng)
        pts = rng.normal(0, 4, (n, 3)).astype(np.float32)
        pts[rng.random(n) < 0.3, 1] = np.nan
        d = [torch.from_numpy(parts.copy()).cuda(), torch.from_numpy(pts).cuda(), torch.zeros(6, device="cuda")]
        want = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        keep.append((parts, d, want))
        filters.append({"map": dmap, "P": P, "N": n, "tf": synth.IDENTITY_TF, "particles": d[0].data_ptr(),
                        "points": d[1].data_ptr(), "pose_out": d[2].data_ptr()})
    torch.cuda.synchronize()
    b = FilterBatch(ctx, filters)
    if captured:
        b.capture()
    for tiles in ((1024, 2), (64, 1)):
        b.set_tiles(*tiles)
        for _ in range(4):
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
    ctx.close()
