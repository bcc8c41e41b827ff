"""Calls of different sizes from several threads at once: a kernel's shared-memory
limit is process state, so no thread's small frame may take it away between another
thread's setting and its launch.  Frames whose kernels need from a few kilobytes to
the most shared memory they use."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-40.0, 40.0, (3 * n + 50, 3))
    return x[np.linalg.norm(x, axis=1) > 3.0][:n], rng.normal(0.0, 0.4, n)


def _at_once(calls, repeats):
    want = [c() for c in calls]
    errors = []

    def loop(call, w):
        try:
            for _ in range(repeats):
                np.testing.assert_array_equal(call(), w)
        except Exception as e:  # reported below
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(c, w)) for c, w in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:2]


def test_point_fields(gpu_lib):
    from pycpet_gb300 import esp_grid, field_grid

    calls = []
    for n in (200, 32000, 700, 16000, 2500, 32000):
        x, q = _frame(n, n)
        pts = np.random.default_rng(n).uniform(-1.0, 1.0, (1, 3))
        calls.append(lambda x=x, q=q, p=pts: field_grid(p, x, q, clamp=False))
        calls.append(lambda x=x, q=q, p=pts: esp_grid(p, x, q))
    _at_once(calls, 400)


@pytest.mark.parametrize("lines", [20, 16 * 200])  # team kernel; persistent kernel and hand-over
def test_streamlines(gpu_lib, lines):
    from pycpet_gb300 import topo_lines

    calls = []
    for n in (60, 12000, 300, 12000):
        x, q = _frame(n, n)
        starts = np.random.default_rng(n).uniform(-1.2, 1.2, (lines, 3))
        caps = np.full(lines, 8, np.int32)
        calls.append(lambda a=(starts, caps, x, q): topo_lines(*a, 0.05, [1.5, 1.5, 1.2]))
    _at_once(calls, 300)
