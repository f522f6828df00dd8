"""The motion update's and the pose kernel's float-pair trigonometry on the GPU:
bit for bit the double functions' roundings, over ordinary values and those the
pairs leave to the double functions (zeros of both signs, tiny, huge and
non-finite draws, angles beyond the reduction's range, gimbal lock)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context, MotionModel
from tsdf_localization_gb300 import _native as N

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def particles(P, seed, spread):
    rng = np.random.default_rng(seed)
    p = np.zeros((P, 7), np.float32)
    p[:, :3] = rng.uniform(-80, 80, (P, 3))
    p[:, 3:6] = rng.uniform(-spread, spread, (P, 3))
    p[:, 6] = rng.random(P)
    return p


def bits(a):
    return np.where(np.isnan(a), np.float32(np.nan), a).view(np.uint32)


@pytest.mark.parametrize("spread", [0.0, 1e-6, 0.1, np.pi, 63.9, 1e4])
@pytest.mark.parametrize("P", [1, 127, 129, 60_000])
def test_given_draws(ctx, P, spread):
    parts = particles(P, 5, spread)
    rng = np.random.default_rng(6)
    draws = rng.normal(0, [0.4, 0.1, 0.05, 0.08, 0.08, 0.6], (P, 6))
    odd = np.array([0.0, -0.0, 1e-30, -1e-19, 1e-300, 0.25, np.pi / 2, -np.pi, 63.0, 70.0, 1e12, 0.1])
    rows = rng.random(P) < 0.3
    draws[rows] = odd[rng.integers(0, odd.size, (int(rows.sum()), 6))]
    parts[rng.random(P) < 0.1, 3:6] = np.float32([-0.0, np.pi / 2, 0.0])
    got = MotionModel(ctx).apply(parts.copy(), draws)
    assert np.array_equal(bits(got), bits(O.motion_apply(parts, draws)))


@pytest.mark.parametrize("mean,sd", [
    ([0.1, 0, 0, 0, 0, 0.02], [0.4, 0.1, 0.05, 0.08, 0.08, 0.6]),
    ([0.1, 0, 0, 0, 0, 0.02], [0.1, 0.1, 0, 0, 0, 0.1]),          # planar: no draw in three axes
    ([0, 0, 0, 0, 0, 0], [0, 0, 0, 0, 0, 0]),
    ([1e-25, -0.0, 3e11, 1e-3, -2.0, 50.0], [0.1, 1e-21, 1e11, 0.1, 0.3, 20.0]),   # beyond the pairs' range
    ([-5.0, 2.0, 1.0, 0.3, 0.2, 3.0], [1e-6, 3.0, 1e-3, 1e-7, 2.0, 1e-12]),
])
@pytest.mark.parametrize("P", [1, 1000, 100_001])
def test_generated_draws_compose_as_the_same_draws_given(ctx, mean, sd, P):
    parts = particles(P, 8, np.pi)
    m = N.Motion((C.c_double * 6)(*mean), (C.c_double * 6)(*sd))
    with_draws, alone = torch.from_numpy(parts).cuda(), torch.from_numpy(parts).cuda()
    d_draws = torch.zeros((P, 6), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for d_part, d_out in ((with_draws, d_draws.data_ptr()), (alone, None)):
        N.check(N.lib().tsdfl_motion_update_device(ctx.handle, C.c_void_p(d_part.data_ptr()), P, C.byref(m), 17, 4,
                                                   C.c_void_p(d_out)))
    ctx.sync()
    want, got, draws = with_draws.cpu().numpy(), alone.cpu().numpy(), d_draws.cpu().numpy()
    assert np.array_equal(bits(got), bits(want))
    assert np.array_equal(bits(want), bits(O.motion_apply(parts, draws)))
