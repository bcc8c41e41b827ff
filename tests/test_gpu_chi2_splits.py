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
