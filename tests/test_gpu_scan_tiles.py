"""Scan reduction at its tiles' edges (1,024 points) and where the prefix kernels
come in (beyond 256 tiles), against the oracle: the same points in the same order,
bit for bit; clouds with few and with all 64 rings, most points dropped, and
outputs that do not hold every point."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context, ScanReducer, pack_cloud
from tsdf_localization_gb300 import _native as N

pytestmark = pytest.mark.gpu
TILE, DIRECT = 1024, 256 * 1024


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def cloud(n, rings, near, seed):
    rng = np.random.default_rng(seed)
    xyz = rng.normal(0, 6, (n, 3)).astype(np.float32)
    xyz[rng.random(n) < near] *= np.float32(0.01)
    return xyz, rng.integers(0, rings, n).astype(np.int16)


@pytest.mark.parametrize("own_ring", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, TILE - 1, TILE, TILE + 1, 3 * TILE + 7, DIRECT - 1, DIRECT, DIRECT + 1,
                               DIRECT + 5 * TILE + 3, 1_200_001])
@pytest.mark.parametrize("rings,near", [(64, 0.1), (1, 0.0), (33, 0.95)])
def test_tile_edges(ctx, n, rings, near, own_ring):
    xyz, ring = cloud(n, rings, near, n + rings)
    for _ in range(2):   # the second finds the first's table and counts
        got = ScanReducer(ctx, 0.3, own_ring).reduce_xyz(xyz, ring)
        assert np.array_equal(got, O.reduce_scan(xyz, ring, 0.3, own_ring))


@pytest.mark.parametrize("n", [5000, DIRECT + 5000])
def test_output_of_too_few_points(ctx, n):
    xyz, ring = cloud(n, 64, 0.1, 9)
    blob, out, cnt = pack_cloud(xyz, ring), np.zeros((700, 3), np.float32), C.c_size_t(0)
    rc = N.lib().tsdfl_reduce_scan(ctx.handle, blob.ctypes.data, n, 16, 0, 12, 0.3, 0, out.ctypes.data, 700,
                                   C.byref(cnt))
    want = O.reduce_scan(xyz, ring, 0.3)
    assert rc == N.TSDFL_ERR_CAPACITY and cnt.value == want.shape[0] and np.array_equal(out, want[:700])
