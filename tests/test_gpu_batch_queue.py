"""The batch's scoring queue (items of every segment from the segment's own
counter) and its filters' kernels side by side: more segments than a warp has
lanes, more segments than items a warp, one filter alone, few items for many
multiprocessors; filters that share buffers run in their order; the first
filter's device error is the one reported.  Every filter's results equal its
single-filter results bit for bit."""
import numpy as np
import pytest

from tsdf_localization_gb300 import FilterBatch
from tsdf_localization_gb300 import _native as N

from test_gpu_batch import check_same, ctx, make_filters, maps, single  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = {
    "one item": [(1, 1)],
    "one filter": [(700, 3000)],
    "segments beyond a warp's lanes": [(3 + 5 * i, 1 + 37 * i) for i in range(75)],
    "one large among small": [(2, 65)] * 20 + [(9000, 3001)] + [(5, 1023), (6, 1024), (7, 1025)] * 4,
    "two passes": [(600, 21_000), (50, 64), (900, 17_000)],
}


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("shape", [(1024, 2), (64, 1), (2048, 8)])
@pytest.mark.parametrize("name", list(SIZES))
def test_queue_equals_single_filters(ctx, maps, name, shape, captured):  # noqa: F811
    fs, keep = make_filters(maps[:4], SIZES[name], 40)
    b = FilterBatch(ctx, fs)
    N.check(N.lib().tsdfl_batch_set_tiles(b.handle, *shape))
    if captured:
        b.capture()
    for _ in range(2):
        for k in keep:
            k["part"].copy_(torch.from_numpy(k["parts0"]))
        torch.cuda.synchronize()
        b.run()
        ctx.sync()
        check_same(ctx, keep, SIZES[name])
    b.close()


@pytest.mark.parametrize("captured", [False, True])
def test_filters_sharing_buffers_run_in_their_order(ctx, maps, captured):  # noqa: F811
    sizes = [(400 + i, 300) for i in range(9)]
    fs, keep = make_filters(maps[:4], sizes, 60)
    last = keep[-1]
    for f in fs[:-1]:   # all write the last one's outputs
        f.update(resampled=last["out"].data_ptr(), count=last["cnt"].data_ptr(), pose_out=last["pose"].data_ptr())
    b = FilterBatch(ctx, fs)
    if captured:
        b.capture()
    torch.cuda.synchronize()
    for _ in range(5):
        last["out"].zero_()
        for k in keep:
            k["part"].copy_(torch.from_numpy(k["parts0"]))
        torch.cuda.synchronize()
        b.run()
        ctx.sync()
        check_same(ctx, [last], sizes[-1:])
        for k, (P, _) in zip(keep[:-1], sizes):
            assert np.array_equal(k["part"].cpu().numpy(), single(ctx, k, P)[0])
    b.close()


def test_a_filters_device_error_is_reported(ctx, maps):  # noqa: F811
    sizes = [(500, 200)] * 6
    fs, keep = make_filters(maps[:4], sizes, 80)
    fs[3]["cap"] = 1   # its resampler emits more than fit
    b = FilterBatch(ctx, fs)
    torch.cuda.synchronize()
    b.run()
    with pytest.raises(N.TsdflError):
        ctx.sync()
    check_same(ctx, [k for i, k in enumerate(keep) if i != 3], sizes[:5])
    b.close()
