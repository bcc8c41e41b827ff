"""The team kernel (few lines per SM, and the last lines of larger launches)
against the persistent kernel: a line's sums and their order are the same in
both, so its result is the same bits whether it runs in a launch of a few lines
(teams from the start), of a few hundred (teams in several rounds) or of
thousands (persistent kernel, then hand-over).  Frame sizes at the edges of a
Kahan run (2,048 charges; 512 sources in FP64), of the teams' shared memory and
of the persistent kernel's; line counts at the edges of the choice (16 lines
per SM, one line per SM)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-40.0, 40.0, (3 * n + 50, 3))
    x = x[np.linalg.norm(x, axis=1) > 3.0][:n]
    return x, rng.normal(0.0, 0.4, n), rng.normal(0.0, 0.3, (n, 3))


def _lines(L, seed):
    rng = np.random.default_rng(seed)
    starts = rng.uniform(-1.5, 1.5, (L, 3))
    caps = rng.integers(0, 400, L).astype(np.int32)
    caps[:6] = [0, 1, 2, 3, -4, 400]
    return starts, caps


def _run(dipoles, starts, caps, x, src, step, precision):
    from pycpet_gb300 import topo_dipole_lines, topo_lines

    fn = topo_dipole_lines if dipoles else topo_lines
    return fn(starts, caps, x, src, step, [1.5, 1.5, 1.2], precision=precision, return_ends=True, return_steps=True)


@pytest.mark.parametrize("dipoles", [False, True])
@pytest.mark.parametrize("precision,n", [("fp32c", 1), ("fp32c", 65), ("fp32c", 2048), ("fp32c", 2049),
                                         ("fp32c", 8000), ("fp32c", 12737), ("fp32c", 20000), ("fp64", 1),
                                         ("fp64", 512), ("fp64", 513), ("fp64", 1500)])
def test_few_lines_equal_many(gpu_lib, precision, n, dipoles):
    x, q, mu = _frame(n, n + 7)
    src = mu if dipoles else q
    step = 0.01 if precision == "fp32c" else 0.02
    L = 16 * gpu_lib.cpetgb_device_sms() + 1          # one more than the teams take at once
    starts, caps = _lines(L, n)
    many = _run(dipoles, starts, caps, x, src, step, precision)
    sms = gpu_lib.cpetgb_device_sms()
    # 1 .. 16 lines per SM: every number of lines a team can hold
    for k in [1, 7, sms, sms + 1, L - 1] + [sms * m for m in range(2, 16)]:
        few = _run(dipoles, starts[:k], caps[:k], x, src, step, precision)
        for a, b in zip(few, many):
            np.testing.assert_array_equal(a, b[:k])


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_batches_of_few_and_many_lines(gpu_lib, precision):
    """Frames with and without lines, more frames than a warp scans at once, in
    launches on both sides of the choice, directly and as plans."""
    import torch
    from pycpet_gb300 import TopoBatch, synchronize

    sizes = (300, 2049, 900, 13000 if precision == "fp32c" else 600)
    frames = [_frame(n, n) for n in sizes]

    def batch(line_counts):
        out = []
        for i, L in enumerate(line_counts):
            x, q, _ = frames[i % len(frames)]
            starts, caps = _lines(max(L, 6), 50 + i)
            out.append({"x": x, "q": q, "starts": starts[:L], "n_iter": caps[:L], "step": 0.01 + 0.01 * (i % 2),
                        "half_dims": [1.5, 1.5, 1.2]})
        return out

    for counts in ([3, 0, 40, 1], [5] * 41, [900, 0, 1300, 700], [80] * 37):
        fr = batch(counts)
        res, steps = TopoBatch(fr, precision=precision).run(return_steps=True)
        plan = TopoBatch(fr, precision=precision, device=True, graph=True)
        for _ in range(2):  # a replay starts from zeroed counters again
            pr, ps = plan.run(return_steps=True)
        synchronize()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(pr.cpu().numpy(), res)
        np.testing.assert_array_equal(ps.cpu().numpy(), steps)
        off = 0
        for f in fr:
            L = len(f["starts"])
            if L:
                one = _run(False, f["starts"], f["n_iter"], f["x"], f["q"], f["step"], precision)
                np.testing.assert_array_equal(res[off:off + L], one[0])
                np.testing.assert_array_equal(steps[off:off + L], one[2])
            off += L
