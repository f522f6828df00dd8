"""The parallel residual systematic resampler against the oracle's serial chain:
indices and counts bit for bit at the edges of its tiles and size classes, for
weights that keep the chain inside the candidate windows and weights that do
not (zeros, a few large weights, heavy tails)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context, ResidualSystematicResampler
from tsdf_localization_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def weights(kind: str, m: int, rng) -> np.ndarray:
    w = {"even": lambda: np.ones(m), "uneven": lambda: 0.02 + rng.gamma(0.8, size=m),
         "flat": lambda: np.exp(rng.normal(0, 0.05, m)), "tail": lambda: np.exp(rng.normal(0, 3, m)),
         "sparse": lambda: np.where(rng.random(m) < 40.0 / m, rng.random(m), 0.0),
         "scaled": lambda: 2.5 + 0.3 * rng.random(m)}[kind]()
    if kind == "sparse":
        w[m // 2] = 1.0
    # "scaled" weights sum to 2.5: about 2.5 outputs a particle, as unnormalised weights give
    return (w / w.sum() * (2.5 if kind == "scaled" else 1.0)).astype(np.float32)


@pytest.mark.parametrize("kind", ["even", "uneven", "flat", "tail", "sparse", "scaled"])
@pytest.mark.parametrize("m", [2559, 2560, 2561, 4096, 4609, 23457, 262143, 262145, 1048577])
def test_matches_serial_chain(ctx, m, kind):
    rng = np.random.default_rng(m + len(kind))
    w = weights(kind, m, rng)
    for u0 in (0.0, 0.371, float(np.nextafter(np.float32(1.0), np.float32(0)))):
        got = ResidualSystematicResampler(ctx).resample_indices(w, u0, cap=4 * m + 16)
        assert np.array_equal(got, O.resample_residual_systematic(w, u0, cap=4 * m + 16))


def test_particles_capacity_and_bad_weights(ctx):
    """The device form's copies; an output buffer that is too small (the count
    still complete, nothing written past it); a negative weight far into the cloud."""
    torch = pytest.importorskip("torch")
    m = 30_000
    rng = np.random.default_rng(5)
    p = rng.normal(size=(m, 7)).astype(np.float32)
    p[:, 6] = weights("uneven", m, rng)
    idx = O.resample_residual_systematic(p[:, 6].copy(), 0.25, cap=2 * m)
    d_in = torch.from_numpy(p).cuda()

    def call(d, cap):
        out = torch.full((idx.shape[0] + 8, 7), -1.0, device="cuda")
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        N.check(N.lib().tsdfl_resample_residual_systematic_device(
            ctx.handle, C.c_void_p(d.data_ptr()), m, 0.25, C.c_void_p(out.data_ptr()), cap,
            C.c_void_p(cnt.data_ptr())))
        rc = N.lib().tsdfl_ctx_sync(ctx.handle)
        return rc, out.cpu().numpy(), int(cnt.item())

    rc, out, n = call(d_in, idx.shape[0])
    assert rc == N.TSDFL_OK and n == idx.shape[0] and np.array_equal(out[:n], p[idx])
    rc, out, n = call(d_in, 10_001)
    assert rc == N.TSDFL_ERR_CAPACITY and n == idx.shape[0]
    assert np.array_equal(out[:10_001], p[idx[:10_001]]) and np.all(out[10_001:] == -1.0)
    bad = d_in.clone()
    bad[29_000, 6] = -1.0
    rc, out, n = call(bad, idx.shape[0])
    assert rc == N.TSDFL_ERR_UNSUPPORTED and np.all(out == -1.0)
    rc, out, n = call(d_in, idx.shape[0])
    assert rc == N.TSDFL_OK and np.array_equal(out[:n], p[idx])
