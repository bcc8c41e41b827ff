"""The FP64 pair weights q / r^3 and q / r (integer-built powers of a MUFU seed
inside r^2 = 2^-100 .. 2^100, the plain form outside) against Coulomb's law in
extended precision, over distances on both sides of that range and next to
powers of two.

Tolerance: 1.2e-15 relative.  The weight is off by at most 3.8 units of 2^-53
inside the range and 5.5 outside, r^2 by one (x 1.5), the products with the
component and with the Coulomb constant by one each: 10 units, 1.1e-15."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = np.longdouble(14.3996451)
TOL = 1.2e-15


def _distances():
    r = [np.float64(2.0) ** e for e in range(-60, 61)]
    r += [np.nextafter(2.0 ** e, 0.0) for e in range(-60, 61, 4)]
    r += [np.nextafter(2.0 ** e, np.inf) for e in range(-60, 61, 4)]
    rng = np.random.default_rng(1)
    r += list(2.0 ** rng.uniform(-60, 60, 600)) + list(rng.uniform(0.5, 80.0, 1200))
    return np.array(r)


@pytest.mark.parametrize("device", [False, True])
def test_single_pairs(gpu_lib, device):
    from pycpet_gb300 import esp_grid, field_grid

    r = _distances()
    pts = np.zeros((len(r), 3))
    pts[:, 1] = r
    x, q = np.zeros((1, 3)), np.array([0.7310585])
    if device:
        import torch

        pts, x, q = (torch.from_numpy(a).cuda() for a in (pts, x, q))
    E = field_grid(pts, x, q, precision="fp64", clamp=False)
    phi = esp_grid(pts, x, q, precision="fp64")
    if device:
        E, phi = E.cpu().numpy(), phi.cpu().numpy()
    rl = r.astype(np.longdouble)
    ql = np.longdouble(0.7310585)
    ref = K * ql / (rl * rl)
    assert np.all(E[:, [0, 2]] == 0.0)
    assert np.abs((E[:, 1] - ref) / ref).max() <= TOL
    assert np.abs((phi - K * ql / rl) * rl / (K * ql)).max() <= TOL


def test_coincident_and_nonfinite(gpu_lib):
    """A point on a charge, an infinite and a NaN coordinate: the plain form's
    values (infinite potential, NaN field without the clamp)."""
    from pycpet_gb300 import esp_grid, field_grid

    pts = np.array([[0.0, 0, 0], [1.0, 0, 0], [np.inf, 0, 0], [np.nan, 0, 0]])
    x, q = np.zeros((1, 3)), np.array([1.0])
    phi = esp_grid(pts, x, q, precision="fp64")
    assert np.isposinf(phi[0]) and phi[2] == 0.0 and np.isnan(phi[3])
    E = field_grid(pts, x, q, precision="fp64", clamp=False)
    assert np.isnan(E[0]).all() and np.isnan(E[2, 0]) and np.isnan(E[3]).any()
    assert E[2, 1] == 0.0 and E[2, 2] == 0.0
    E = field_grid(pts[:2], x, q, precision="fp64", clamp=True)
    assert np.all(E[0] == 0.0)
    np.testing.assert_allclose(E[1], [14.3996451, 0, 0], rtol=1e-15)
