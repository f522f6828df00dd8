"""A filter that fills the GPU by itself with a cloud spread over the map, among
small ones: its particles are put in spatial order inside the batch's update, and
the autotuner scores the same poses many times over.  Every filter's results equal
its single-filter results bit for bit, before and after."""
import numpy as np
import pytest

from tsdf_localization_gb300 import FilterBatch

from test_gpu_batch import check_same, ctx, make_filters, maps  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sizes", [[(300, 500), (100_000, 600), (70, 65)], [(90_001, 1100), (84_000, 700), (5, 64)]])
def test_autotune_with_spread_filters(ctx, maps, sizes):  # noqa: F811
    fs, keep = make_filters(maps[:4], sizes, 90)
    rng = np.random.default_rng(9)
    spread = 0
    for k, (P, n) in zip(keep, sizes):
        if P * n < 3 << 24:
            continue
        k["parts0"][:, :2] += rng.uniform(-8, 8, (P, 2)).astype(np.float32)
        spread += 1
    b = FilterBatch(ctx, fs)
    assert spread and b.info()["single"] == spread

    def run_and_check():
        for k in keep:
            k["part"].copy_(torch.from_numpy(k["parts0"]))
        torch.cuda.synchronize()
        b.run()
        ctx.sync()
        check_same(ctx, keep, sizes)

    run_and_check()
    chunk, group, ms = b.autotune()
    assert chunk % 64 == 0 and group >= 1 and 0 < ms < 100
    run_and_check()
    b.capture()
    run_and_check()
    b.close()
