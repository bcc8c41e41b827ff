"""Launches on both sides of the choice between the team kernel (from the start
points, in rounds) and the persistent kernel: the same bits, every line once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-40.0, 40.0, (3 * n + 50, 3))
    return x[np.linalg.norm(x, axis=1) > 3.0][:n], rng.normal(0.0, 0.4, n), rng.normal(0.0, 0.3, (n, 3))


def _lines(L, cap, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1.2, 1.2, (L, 3)), rng.integers(0, cap, L).astype(np.int32)


# FP32C: the limit is 20 lines per SM for sources in shared memory, 32 beyond
@pytest.mark.parametrize("dipoles", [False, True])
@pytest.mark.parametrize("n,per_sm", [(300, (17, 20)), (16000, (17, 31, 32))])
def test_fp32c_limits(gpu_lib, n, per_sm, dipoles):
    from pycpet_gb300 import topo_dipole_lines, topo_lines

    sms = gpu_lib.cpetgb_device_sms()
    x, q, mu = _frame(n, n)
    fn, src = (topo_dipole_lines, mu) if dipoles else (topo_lines, q)
    starts, caps = _lines(sms * per_sm[-1] + 1, 300, 3)
    args = dict(step=0.01, half_dims=[1.5, 1.5, 1.2], return_ends=True, return_steps=True)
    many = fn(starts, caps, x, src, **args)           # one past the limit: persistent
    for k in [sms * m for m in per_sm]:
        for a, b in zip(fn(starts[:k], caps[:k], x, src, **args), many):
            np.testing.assert_array_equal(a, b[:k])


# FP64: the limit is the hand-over records of a launch
@pytest.mark.parametrize("step", [0.02, 0.3])  # several rounds, one round
def test_fp64_limit(gpu_lib, step):
    from pycpet_gb300 import topo_lines

    L = (1 << 18) + 1
    x, q, _ = _frame(33, 5)
    starts, caps = _lines(L, 6, 4)
    caps[::5000] = 400
    args = dict(precision="fp64", return_ends=True, return_steps=True)
    many = topo_lines(starts, caps, x, q, step, [1.5, 1.5, 1.2], **args)  # persistent
    for lo, hi in [(0, L - 1), (0, 40000), (L - 2433, L)]:
        for a, b in zip(topo_lines(starts[lo:hi], caps[lo:hi], x, q, step, [1.5, 1.5, 1.2], **args), many):
            np.testing.assert_array_equal(a, b[lo:hi])
