"""Systematic resampling against the oracle at the edges of its tiles, chunks
and blocks, on every path: exact fixed-point sums, chained double sums (weights
below 2^-29, starting with zeros, crossing binades inside and between chunks) and
the literal loop (a negative weight); twice each, since the kernels' block
counters have to be clear for the next call."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context, SystematicResampler

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def weights(kind: str, m: int, rng) -> np.ndarray:
    w = rng.random(m) + 0.01
    if kind == "small":      # many weights that are no multiples of 2^-52
        w = w ** 6 * 1e-4
        w[rng.integers(0, m, max(1, m // 50))] = 1.0
        w[: m // 3] *= 1e-12
    if kind == "zeros":
        w[: m // 2] = 0.0
        w[m // 2:] **= 8
    if kind == "halves":     # total 2 and above: the fixed-point sums leave their range
        return (w / w.sum() * 2.5).astype(np.float32)
    w = (w / w.sum()).astype(np.float32)
    if kind == "negative":
        w[m // 2] = -w[m // 2] / 8
    return w


@pytest.mark.parametrize("kind", ["even", "small", "zeros", "halves", "negative"])
@pytest.mark.parametrize("m", [1, 2, 63, 64, 65, 1023, 1024, 1025, 4096, 4097, 32_769, 131_073, 140_000])
def test_matches_serial_loop(ctx, m, kind):
    rng = np.random.default_rng(m * 5 + len(kind))
    w = weights(kind, m, rng)
    rs = SystematicResampler(ctx)
    for u in (0.0, 0.37, 0.999):
        u0 = float(np.float32(u / m))
        got = rs.resample_indices(w, u0, cap=3 * m + 16)
        assert np.array_equal(got, O.resample_systematic(w, u0, cap=3 * m + 16)), (m, kind, u)
