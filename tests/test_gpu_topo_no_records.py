"""Streamline launches without memory for hand-over records (one round, no hand-over):
the bits of the launch with them, for single frames on both sides of the kernels'
limits, for tables and for replayed plans."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def records(gpu_lib):
    yield gpu_lib.cpetgb_set_hand_over_records
    gpu_lib.cpetgb_set_hand_over_records(1)


def _frame(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-40.0, 40.0, (3 * n + 50, 3))
    return x[np.linalg.norm(x, axis=1) > 3.0][:n], rng.normal(0.0, 0.4, n), rng.normal(0.0, 0.3, (n, 3))


def _lines(L, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1.2, 1.2, (L, 3)), rng.integers(0, 300, L).astype(np.int32)


# 2 to 20 lines per SM: team kernel in FP64 and for 12,800 sources; 40: persistent kernel
# with hand-over for those; 600 sources in FP32C: never either
@pytest.mark.parametrize("dipoles", [False, True])
@pytest.mark.parametrize("precision,n,step", [("fp32c", 600, 0.01), ("fp32c", 12800, 0.01), ("fp32c", 12800, 0.3),
                                              ("fp64", 600, 0.01), ("fp64", 600, 0.3)])
def test_single_frames(records, precision, n, step, dipoles):
    from pycpet_gb300 import _lib, topo_dipole_lines, topo_lines

    sms = _lib.device_sms()
    x, q, mu = _frame(n, 3)
    fn, src = (topo_dipole_lines, mu) if dipoles else (topo_lines, q)
    for per_sm in (2, 16, 17, 20, 21, 40):
        starts, caps = _lines(sms * per_sm, per_sm)
        run = lambda: fn(starts, caps, x, src, step, [1.5, 1.5, 1.2], precision=precision, return_ends=True,
                         return_steps=True)
        assert records(1) == 0
        want = run()
        assert records(0) == 0
        for a, b in zip(run(), want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision,sizes", [("fp32c", (300, 13900, 12800)), ("fp64", (300, 2049, 700))])
@pytest.mark.parametrize("counts", [[3, 0, 40, 1], [900, 0, 1300, 700], [3000, 5, 2500]])
def test_tables_and_plans(records, precision, sizes, counts):
    import torch
    from pycpet_gb300 import TopoBatch

    frames = []
    for i, L in enumerate(counts):
        x, q, _ = _frame(sizes[i % 3], i)
        starts, caps = _lines(max(L, 1), 40 + i)
        frames.append({"x": x, "q": q, "starts": starts[:L], "n_iter": caps[:L], "step": 0.01 + 0.01 * (i % 2),
                       "half_dims": [1.5, 1.5, 1.2]})
    want = TopoBatch(frames, precision=precision).run(return_steps=True)
    assert records(0) == 0
    for a, b in zip(TopoBatch(frames, precision=precision).run(return_steps=True), want):
        np.testing.assert_array_equal(a, b)
    plan = TopoBatch(frames, precision=precision, device=True, graph=True)
    assert records(1) == 0
    for _ in range(2):
        got = plan.run(return_steps=True)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a.cpu().numpy(), b)


def test_the_setting_is_the_threads_own(records):
    """Another thread's calls keep their records (the same results either way)."""
    import threading

    from pycpet_gb300 import topo_lines

    x, q, _ = _frame(12800, 4)
    starts, caps = _lines(5000, 5)
    want = topo_lines(starts, caps, x, q, 0.01, [1.5, 1.5, 1.2])
    assert records(0) == 0
    got = []
    t = threading.Thread(target=lambda: got.append(topo_lines(starts, caps, x, q, 0.01, [1.5, 1.5, 1.2])))
    t.start()
    here = topo_lines(starts, caps, x, q, 0.01, [1.5, 1.5, 1.2])
    t.join()
    np.testing.assert_array_equal(got[0], want)
    np.testing.assert_array_equal(here, want)
