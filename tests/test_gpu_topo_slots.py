"""Launches that fill a CTA's line slots more than once, on both sides of the rule on
their number (1,024 sources, 96 lines per SM) and with either tuned number: the same
bits, single frames and tables."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 1024, 1025])
def test_slots(gpu_lib, n):
    from pycpet_gb300 import TopoBatch, topo_lines

    L = 97 * gpu_lib.cpetgb_device_sms()
    rng = np.random.default_rng(n)
    x = rng.uniform(-40.0, 40.0, (2 * n + 20, 3))
    x = x[np.linalg.norm(x, axis=1) > 3.0][:n]
    q = rng.normal(0.0, 0.4, n)
    starts, caps = rng.uniform(-1.2, 1.2, (L, 3)), rng.integers(0, 60, L).astype(np.int32)
    half = [1.5, 1.5, 1.2]
    keys = [gpu_lib.cpetgb_tune_key(1, 1, c, float(s)) for c in (0, 1) for s in (500, 3000, 9000, 20000, 70000)]
    before = [gpu_lib.cpetgb_tune_get(k) for k in keys]
    got = []
    try:
        for v in (0, 1):
            for k in keys:
                assert gpu_lib.cpetgb_tune_set(k, v) == 0
            for m in (L, L - gpu_lib.cpetgb_device_sms() - 1):
                got.append(topo_lines(starts[:m], caps[:m], x, q, 0.02, half, return_steps=True))
            frame = {"x": x, "q": q, "starts": starts, "n_iter": caps, "step": 0.02, "half_dims": half}
            r, s = TopoBatch([frame, frame], precision="fp32c").run(return_steps=True)
            got += [(r[:L], s[:L]), (r[L:], s[L:])]
    finally:
        for k, v in zip(keys, before):
            gpu_lib.cpetgb_tune_set(k, v)
    for r, s in got:
        np.testing.assert_array_equal(r, got[0][0][: len(r)])
        np.testing.assert_array_equal(s, got[0][1][: len(s)])
