"""The FP32C chi-square kernels at the edges of their tiles, chunks and splits.

Bound for rows that sum to 1 (D <= 1), u = 2^-24: rounding the two values moves a
term (a-b)^2/(a+b) by at most 2 u (a+b), its own operations (the MUFU reciprocal's
1 ulp included) by 5 u, a chunk's plain sum by 31 u; the Kahan sums of chunks and
splits add 2 u.  Over a row pair sum(a+b) = 2, halved: at most (4 + 5 + 31 + 2) u."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 42 * 2.0 ** -24


# one row; a block exactly and one past it; a chunk exactly and one past it; bins at
# which the splits begin (256) and end raggedly; enough tiles for a single split
@pytest.mark.parametrize("n,bins", [(1, 300), (64, 1), (65, 32), (128, 33), (127, 256), (129, 257), (64, 901),
                                    (200, 95), (700, 391), (2300, 259)])
def test_against_float64(gpu_lib, n, bins):
    import torch
    from pycpet_gb300 import chi2_distance_matrix

    rng = np.random.default_rng(n * 1000 + bins)
    h = rng.random((n, bins)) * (rng.random((n, bins)) < 0.4)
    h[0, 0] = 1.0
    h[n // 2] = 0.0
    if n > 3:
        h[3] = h[1]
    s = h.sum(axis=1, keepdims=True)
    h = np.divide(h, s, out=np.zeros_like(h), where=s > 0)
    d = chi2_distance_matrix(h, "fp32c")
    t = torch.from_numpy(h).cuda()
    ref = np.empty((n, n))
    for i in range(n):
        sm, df = t + t[i], t - t[i]
        ref[i] = (0.5 * torch.where(sm != 0, df * df / torch.where(sm != 0, sm, 1.0), 0.0).sum(1)).cpu().numpy()
    np.testing.assert_allclose(d, ref, rtol=0, atol=BOUND)
    np.testing.assert_array_equal(d, d.T)
    assert np.all(np.diag(d) == 0)
    if n > 3:
        assert d[1, 3] == 0.0


def test_signed_zeros_negatives_and_non_finite_values(gpu_lib):
    """Whatever a bin holds, the value is the definition's: empty pairs of either
    sign contribute nothing, an infinity or NaN gives NaN in its row only."""
    from pycpet_gb300 import chi2_distance_matrix

    h = np.array([[0.5, 0.5, -0.0, 0.0], [0.25, 0.75, -0.0, -0.0], [0.5, -0.25, 0.0, -0.0],
                  [np.inf, 0.5, 0.0, 0.5], [0.5, np.nan, 0.0, 0.5]])
    d = chi2_distance_matrix(h, "fp32c")
    a, b = h[:3, None, :], h[None, :3, :]
    with np.errstate(all="ignore"):
        ref = 0.5 * np.where(a + b != 0, (a - b) ** 2 / (a + b), 0.0).sum(-1)
    np.testing.assert_allclose(d[:3, :3], ref, rtol=1e-6, atol=0)
    assert np.all(np.isnan(d[3:, :3])) and np.all(np.isnan(d[:3, 3:])) and np.all(np.diag(d) == 0)


def test_fp64_quotients_are_the_divisions(gpu_lib):
    """Two rows of one bin each give half a quotient (a - b)^2 / (a + b), compared
    with numpy's division: over sums on both sides of the fast form's range and next
    to powers of two, squares that overflow or vanish.  Tolerance: one unit of 2^-52
    (the sum of one term is exact)."""
    from pycpet_gb300 import chi2_distance_matrix

    rng = np.random.default_rng(5)
    s = [2.0 ** e for e in range(-110, 111, 3)] + [np.nextafter(2.0 ** e, 0.0) for e in range(-110, 111, 7)]
    s += list(2.0 ** rng.uniform(-105, 105, 300)) + list(rng.uniform(1e-6, 2.0, 600)) + [1e-310, 1e308, 3.0]
    s = np.array(s)
    b = s * rng.random(len(s))
    a = s - b
    a[-1], b[-1] = 1e200, -1e200 * (1 - 2.0 ** -50)
    with np.errstate(all="ignore"):
        want = 0.5 * ((a - b) ** 2 / (a + b))
    got = np.array([chi2_distance_matrix(np.array([[x], [y]]), "fp64")[0, 1] for x, y in zip(a, b)])
    np.testing.assert_allclose(got, want, rtol=2.0 ** -52, atol=5e-324)
