"""The subsampling kernel against the oracle: strata stepped without divisions
(every remainder class of N over K, one to three steps of 64 strata, K = 1 and
K = N), scans in shared memory and beyond it, particles taken singly and in
twos, compact and spread clouds.  Hit counts are equal; raw weights are within
1e-5 of the FP64 sums (the fixed-point sum is exact to 2^-30 a point, the one
rounding to float is 2^-24)."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context, DeviceMap, TSDFEvaluator
from tsdf_localization_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def room(ctx):
    wl = synth.room_workload(seed=1, n_particles=10, n_points=2048)
    om = O.OracleMap(O.coef_from(wl.coef), wl.grid_occ, wl.float_data())
    return wl, om, {d: DeviceMap(ctx, wl.coef, wl.grid_occ, codes=wl.codes, dense=d) for d in (True, False)}


def points(wl, n):
    rng = np.random.default_rng(n)
    if n <= wl.points.shape[0]:
        return np.ascontiguousarray(wl.points[:n])
    return np.concatenate([wl.points, rng.normal(0, 5, (n - wl.points.shape[0], 3))]).astype(np.float32)


def check(room, parts, pts, k, seed, dense, sample):
    wl, om, maps = room
    _, raw, hits = TSDFEvaluator(maps[dense]).evaluate_subsampled(parts.copy(), pts, wl.tf, k, seed, debug=True)
    for i in sample:
        idx = O.subsample_indices(seed, int(i), pts.shape[0], k)
        r = O.evaluate(om, np.ascontiguousarray(parts[i:i + 1]).copy(), pts[idx], wl.tf, (0.9, 0.1, 0.0, 100.0), threads=1)
        assert hits[i] == r["hits"][0]
        assert abs(float(raw[i]) - r["sum64"][0]) <= 1e-5 * r["sum64"][0]


@pytest.mark.parametrize("dense", [True, False])
@pytest.mark.parametrize("n,k", [(1, 1), (5, 3), (63, 63), (64, 33), (65, 64), (1000, 65), (1001, 127), (2048, 1),
                                 (2048, 129), (2048, 2048), (9001, 200), (20_011, 193), (40_000, 256)])
def test_strata_and_scan_sizes(room, n, k, dense):
    wl = room[0]
    parts = synth.particles_gaussian(wl.true_pose, 0.3, np.deg2rad(5.0), 70, n + k)
    check(room, parts, points(wl, n), k, 11 + k, dense, range(70))


@pytest.mark.parametrize("P", [1, 31, 5000, 155_647, 156_001])
@pytest.mark.parametrize("spread", [False, True])
def test_particle_counts(room, P, spread):
    wl = room[0]
    parts = synth.particles_gaussian(wl.true_pose, 5.0 if spread else 0.3, np.deg2rad(5.0), P, P)
    sample = np.unique(np.concatenate([np.arange(min(P, 20)), np.arange(max(0, P - 20), P),
                                       np.random.default_rng(P).integers(0, P, 60)]))
    check(room, parts, points(wl, 700), 70, 3, True, sample)
