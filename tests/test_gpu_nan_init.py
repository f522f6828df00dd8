"""A map whose init value is NaN: its fixed-point form (the lowest 64-bit number) leaves
the hit counts and the other values' sums as the generic kernel has them."""
import numpy as np
import pytest

from tsdf_localization_gb300 import Context, DeviceMap, FilterBatch, TSDFEvaluator
from tsdf_localization_gb300 import synth

from test_gpu_scoring_kernels import LAYOUTS, cloud, random_map, scan

pytestmark = pytest.mark.gpu
SIZE = (21.3, 17.6, 5.2)


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def nan_map(ctx, layout):
    coef, occ, codes = random_map(SIZE, 0.1, (0, 0, 0), 1)
    coef.init_value = float("nan")
    return DeviceMap(ctx, coef, occ, codes=codes, sigma=0.1, **LAYOUTS[layout])


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("spread,P,n", [(False, 101, 33), (False, 77, 3001), (True, 395_001, 129)])
def test_hits_and_sums(ctx, layout, spread, P, n):
    rng = np.random.default_rng(P + n)
    dmap = nan_map(ctx, layout)
    parts, pts = cloud(spread, P, SIZE, (0, 0, 0), rng), scan(n, rng)
    fast = TSDFEvaluator(dmap).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
    ref = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
    assert np.array_equal(fast["hits"], ref["hits"]) and np.array_equal(fast["raw"], ref["raw"])
    assert ref["hits"].max() <= n and ref["hits"].min() < n
    if not spread:
        _, raw, hits = TSDFEvaluator(dmap).evaluate_subsampled(parts.copy(), pts, synth.IDENTITY_TF, n, 5, debug=True)
        assert np.array_equal(hits, ref["hits"]) and np.array_equal(raw, ref["raw"])


@pytest.mark.parametrize("layout", ["compact", "brick"])
def test_batched(ctx, layout):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    dmap = nan_map(ctx, layout)
    filters, keep = [], []
    for P, n in ((50, 100), (333, 700), (64, 65)):
        parts, pts = cloud(False, P, SIZE, (0, 0, 0), rng), scan(n, rng)
        want = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        d = [torch.from_numpy(parts.copy()).cuda(), torch.from_numpy(pts).cuda(), torch.zeros(6, device="cuda")]
        keep.append((parts, d, want))
        filters.append({"map": dmap, "P": P, "N": n, "tf": synth.IDENTITY_TF, "particles": d[0].data_ptr(),
                        "points": d[1].data_ptr(), "pose_out": d[2].data_ptr()})
    torch.cuda.synchronize()
    b = FilterBatch(ctx, filters)
    b.run()
    ctx.sync()
    for i, (parts, d, want) in enumerate(keep):
        assert np.array_equal(b.hits(i, parts.shape[0]), want["hits"])
        w = (want["raw"] / np.float32(want["weight_sum"])).astype(np.float32)
        assert np.array_equal(d[0].cpu().numpy()[:, 6], w)
    b.close()
