"""The 8-bit tone map at its steps: the kernel evaluates most values with approximate
reciprocal / log2 / exp2 and must hand every value near a step between bytes, and every
value outside the curve's ordinary range, to the exact formula.  Bytes equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(oracle):
    """The smallest radiance of each byte value, by bisection on the float bits."""
    lo = np.zeros(255, np.int64)
    hi = np.full(255, np.float32(1000.0).view(np.int32), np.int64)
    want = np.arange(1, 256)
    while np.any(hi - lo > 1):
        mid = (lo + hi) // 2
        up = oracle.tonemap(mid.astype(np.int32).view(np.float32)) >= want
        hi, lo = np.where(up, mid, hi), np.where(up, lo, mid)
    return hi


def test_bytes_around_every_step(gpu, oracle):
    bits = (_steps(oracle)[:, None] + np.arange(-300, 301)[None, :]).reshape(-1)
    x = np.concatenate([bits.astype(np.int32).view(np.float32), np.zeros((-len(bits)) % 3, np.float32)])
    assert np.array_equal(gpu.tonemap_aces(x), oracle.tonemap(x))


@pytest.mark.parametrize("n", [3, 6, 15, 4096 * 3, 148 * 8 * 256 * 12 + 3])
def test_lengths_and_special_values(gpu, oracle, n):
    rng = np.random.default_rng(n)
    x = rng.lognormal(-1.0, 2.0, n).astype(np.float32)
    x[rng.integers(0, n, max(1, n // 50))] = rng.choice(
        np.array([0.0, -0.0, -1.0, -1e-30, np.nan, np.inf, -np.inf, 1e-42, 1e19, 3e38, 1e30], np.float32), max(1, n // 50))
    assert np.array_equal(gpu.tonemap_aces(x), oracle.tonemap(x))
