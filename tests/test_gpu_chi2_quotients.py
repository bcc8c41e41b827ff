"""FP64 chi-square terms whose quotient (a - b)^2 / (a + b) lies so close to the middle
between two doubles that a correction by a 24-bit reciprocal rounds it the other way
(found among 2.4e9 random pairs): the division's bits.  One bin per row, so an entry is
half a quotient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAIRS = [("0x1.5213c78cc6dbap-2", "0x1.4bfe6c46baff4p-1"), ("0x1.77c59aa71e401p-1", "0x1.cb7dd675e8474p-3"),
         ("0x1.47699deca96fap-1", "0x1.1c03ab8225de8p-1"), ("0x1.42584301c8771p-1", "0x1.8428ed3c1d7fp-2"),
         ("0x1.023cd0ffdf17p-1", "0x1.2c6bfe9cdd633p-1"), ("0x1.7986cd05b59bcp-2", "0x1.930e084434038p-2"),
         ("0x1.5a060203bf60cp-3", "0x1.0d2aad1bcca8fp-1")]


def test_quotients_next_to_a_middle(gpu_lib):
    from pycpet_gb300 import chi2_distance_matrix

    for a, b in PAIRS:
        a, b = float.fromhex(a), float.fromhex(b)
        d = chi2_distance_matrix(np.array([[a], [b]]), "fp64")
        assert d[0, 1] == d[1, 0] == 0.5 * ((a - b) * (a - b) / (a + b))


def test_random_quotients(gpu_lib):
    """4 million pairs, bit for bit."""
    from pycpet_gb300 import chi2_distance_matrix

    v = np.random.default_rng(3).random(2000) * 2.0 ** np.random.default_rng(4).integers(-20, 20, 2000)
    a, b = v[:, None], v[None, :]
    np.testing.assert_array_equal(chi2_distance_matrix(v[:, None], "fp64"), 0.5 * ((a - b) * (a - b) / (a + b)))
