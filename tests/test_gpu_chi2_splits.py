"""The FP32C chi-square's sums over splits of the bins keep what a double holds: terms
that are powers of two (exact in every step) in different splits, whose sum needs up
to 53 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponents", [(27, 0, -25), (20, -4, -32), (0, -26, -52), (-25, 0, 27), (5, -45, -20, -47)])
@pytest.mark.parametrize("bins", [1024, 20000])
def test_sums_of_powers_of_two(gpu_lib, exponents, bins):
    from pycpet_gb300 import chi2_distance_matrix

    h = np.zeros((2, bins))
    for i, e in enumerate(exponents):       # bins far enough apart for splits of their own
        h[0, (2 * i + 1) * (bins // 10) + i] = 2.0 ** e
    d = chi2_distance_matrix(h, "fp32c")
    want = 0.5 * sum(2.0 ** e for e in sorted(exponents))
    assert d[0, 1] == d[1, 0] == want


# 1 to 6 tiles whose bins are split 15, 16 (the other form of the merge) and 203 ways
@pytest.mark.parametrize("n,bins", [(2, 1000), (64, 1024), (65, 1024), (130, 4200), (100, 20000), (2, 40000)])
def test_many_splits_against_float64(gpu_lib, n, bins):
    """Bound as in test_gpu_chi2.py: 42 x 2^-24 for rows that sum to 1."""
    from pycpet_gb300 import chi2_distance_matrix

    rng = np.random.default_rng(bins + n)
    h = rng.random((n, bins)) * (rng.random((n, bins)) < 0.5)
    h /= h.sum(axis=1, keepdims=True)
    d = chi2_distance_matrix(h, "fp32c")
    ref = np.empty((n, n))
    for i in range(n):
        s = h + h[i]
        ref[i] = 0.5 * np.divide((h - h[i]) ** 2, s, out=np.zeros_like(s), where=s != 0).sum(axis=1)
    np.testing.assert_allclose(d, ref, rtol=0, atol=42 * 2.0 ** -24)
    np.testing.assert_array_equal(d, d.T)
    assert np.all(np.diag(d) == 0)
