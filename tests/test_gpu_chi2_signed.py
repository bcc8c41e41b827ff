"""The FP32C chi-square matrix where histograms hold negative values: a bin whose two
values cancel contributes nothing, as the definition has it, wherever it lies (tile,
chunk of bins, split), and rows without negative values keep their bits.

Tolerance: the values are multiples of 2^-10 below 1, so sums and differences are
exact; with u = 2^-24 a term is off by 5 u (square, MUFU reciprocal, product), a
chunk's plain sum by 31 u, the Kahan sums by 2 u: 38 u of half the terms' magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ref(h):
    a, b = h[:, None, :], h[None, :, :]
    with np.errstate(all="ignore"):
        t = np.where(a + b != 0, (a - b) ** 2 / (a + b), 0.0)
    return 0.5 * t.sum(-1), 0.5 * np.abs(t).sum(-1)


@pytest.mark.parametrize("n,bins", [(2, 1), (3, 33), (70, 64), (65, 401), (130, 901)])
def test_opposite_values_contribute_nothing(gpu_lib, n, bins):
    from pycpet_gb300 import chi2_distance_matrix

    rng = np.random.default_rng(n + bins)
    h = np.round(rng.random((n, bins)) * 1024) / 1024
    plain = chi2_distance_matrix(h, "fp32c")
    g = h.copy()
    g[n - 1, :] = -h[0, :]                       # every bin of the pair (0, n - 1) cancels
    k = bins // 2
    g[0, k], g[n // 2, k] = 0.75, -0.75          # one bin of one pair
    d = chi2_distance_matrix(g, "fp32c")
    ref, mag = _ref(g)
    assert np.all(np.abs(d - ref) <= 38 * 2.0 ** -24 * mag)
    np.testing.assert_array_equal(d, d.T)
    assert np.all(np.diag(d) == 0)
    same = [i for i in range(n) if i not in (0, n // 2, n - 1)]
    np.testing.assert_array_equal(d[np.ix_(same, same)], plain[np.ix_(same, same)])


def test_subnormal_sums(gpu_lib):
    """A sum below the smallest normal float belongs to values whose square vanishes."""
    from pycpet_gb300 import chi2_distance_matrix

    h = np.array([[1e-40, 0.5], [-2e-40, 0.5], [1.5 * 2.0 ** -126, 0.5], [-(2.0 ** -126), 0.5]])
    assert np.all(np.abs(chi2_distance_matrix(h, "fp32c")) <= 1e-37)
