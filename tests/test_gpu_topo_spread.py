"""Tables of frames whose work differs widely: the CTAs start spread over the
frames and move on round the table; every line is done once and has the bits of
a launch of its frame alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a few uneven frames (first, middle and last the heaviest); more frames than CTAs,
# with empty ones at both ends and in runs; a frame past the shared-memory size
@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("sizes", [
    [(3000, 2000), (40, 700), (900, 300)], [(40, 300), (3000, 1800), (500, 500)], [(40, 300), (500, 500), (3000, 1800)],
    [(50, 0), (60, 0)] + [(64 + 7 * (f % 5), (f * 13) % 29) for f in range(260)] + [(30, 0)],
    [(16000, 90), (300, 2500)],
])
def test_every_line_once(gpu_lib, sizes, precision):
    from pycpet_gb300 import TopoBatch, topo_lines
    from pycpet_gb300.synth import make_frame, random_start_points

    if precision == "fp64":
        sizes = [(min(n, 500), L) for n, L in sizes]
    half, step = [0.8, 1.0, 0.9], 0.02
    frames = []
    for f, (n, L) in enumerate(sizes):
        fr = make_frame(n, 100 + f)
        frames.append(dict(starts=random_start_points(max(L, 1), half, 200 + f)[:L], n_iter=40 + f % 7, x=fr["x"],
                           q=fr["q"], step=step, half_dims=half))
    batch = TopoBatch(frames, precision=precision)
    res, steps = batch.run(return_steps=True)
    done = 0
    for fr in frames:
        L = len(fr["starts"])
        if L:
            want, n = topo_lines(fr["starts"], fr["n_iter"], fr["x"], fr["q"], step, half, precision=precision,
                                 return_steps=True)
            np.testing.assert_array_equal(res[done:done + L], want)
            np.testing.assert_array_equal(steps[done:done + L], n)
        done += L
    assert done == len(res)
