"""The float32 host calls (conversions on the GPU) against the double calls with
the same conversions made by numpy: every value is rounded once, so the bits agree."""
import numpy as np
import pytest

from pycpet_gb300 import core, drop_in
from pycpet_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


class _Calc:
    """What the replaced calculator methods read."""

    def __init__(self, x, q, mesh, precision):
        self.x, self.Q, self.mesh = x, q, mesh
        self.precision = precision


def _frame(n, shape, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-20, 20, (n, 3)).astype(np.float32)
    q = rng.uniform(-0.8, 0.8, n).astype(np.float32)
    return x, q, rng.uniform(-3, 3, tuple(shape) + (3,)).astype(np.float32)


# one point; odd counts on both sides of a block of 256; enough points for values
# that two roundings to binary16 would get wrong; more than the staging buffers hold
@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("n,shape", [(1, (1, 1, 1)), (33, (5, 1, 51)), (257, (257, 1, 1)), (500, (41, 41, 41)),
                                     (3, (1300, 1300, 1))])
def test_rows_have_numpys_bits(n, shape, precision):
    x, q, mesh = _frame(n, shape)
    mesh[0, 0, 0] = x[0]  # on a charge: infinities and NaN
    calc = _Calc(x, q, mesh, precision)
    p64, x64, q64 = mesh.reshape(-1, 3).astype(np.float64), x.astype(np.float64), q.astype(np.float64)
    with np.errstate(all="ignore"):
        E = core.field_grid(p64, x64, q64, precision=precision, clamp=True).astype(np.float32)
        phi = core.esp_grid(p64, x64, q64, precision=precision)
        want_half = np.concatenate((mesh.reshape(-1, 3), phi.reshape(-1, 1)), axis=1).astype(np.half)
    got, got_shape = drop_in.compute_box(calc)
    assert got.dtype == np.float32 and got_shape == mesh.shape
    np.testing.assert_array_equal(got, np.concatenate((mesh.reshape(-1, 3), E), axis=1))
    got, got_shape = drop_in.compute_box_ESP(calc)
    assert got.dtype == np.half and got_shape == mesh.shape
    np.testing.assert_array_equal(got, want_half)
    out = np.empty((len(p64), 3), np.float32)
    check(lib().cpetgb_compute_looped_field_p(core.precision_code(precision), len(p64), n, mesh.ctypes.data,
                                              x.ctypes.data, q.ctypes.data, out.ctypes.data))
    np.testing.assert_array_equal(out, E)
    E0 = core.field_grid(np.zeros((1, 3)), x64, q64, precision=precision, clamp=False)[0].astype(np.float32)
    np.testing.assert_array_equal(drop_in.compute_point_field(calc), E0)


def test_other_layouts_and_types_take_the_same_values():
    x, q, mesh = _frame(77, (9, 8, 7))
    want, _ = drop_in.compute_box(_Calc(x, q, mesh, "fp32c"))
    wide = np.zeros((77, 6), np.float32)
    wide[:, ::2] = x
    for a, b, m in [(wide[:, ::2], q, mesh), (np.asfortranarray(x), q, mesh), (x.astype(np.float64), q, mesh),
                    (x, q.astype(np.float64), mesh), (x, q.reshape(-1, 1), mesh), (x, q, np.asfortranarray(mesh))]:
        got, _ = drop_in.compute_box(_Calc(a, b, m, "fp32c"))
        assert got.dtype == np.float32
        np.testing.assert_array_equal(got, want)


def test_threads_have_their_own_buffers():
    from concurrent.futures import ThreadPoolExecutor

    frames = [_frame(50 + 40 * k, (7 + k, 9, 5), seed=k) for k in range(8)]
    calc = [_Calc(*f, "fp32c") for f in frames]
    want = [drop_in.compute_box(c)[0] for c in calc]
    with ThreadPoolExecutor(8) as pool:
        for _ in range(5):
            for got, w in zip(pool.map(lambda c: drop_in.compute_box(c)[0], calc), want):
                np.testing.assert_array_equal(got, w)
