"""Direct device calls recorded into a caller's CUDA graph: replays, long after the call
has returned and its host memory has been used for other things, give the call's bits,
also for new values in the same input tensors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _charges(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-20.0, 20.0, (3 * n, 3))
    return x[np.linalg.norm(x, axis=1) > 3.0][:n], rng.normal(0.0, 0.4, n)


def _record_and_replay(call, tensors, change):
    import torch

    want = call().clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    garbage = [np.full(64 + 16 * k, 0x7FF8DEAD00000000 + k, np.int64) for k in range(4000)]
    out.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    change(*tensors)
    graph.replay()
    got = out.clone()
    torch.cuda.synchronize()
    assert not torch.equal(got, want) and torch.equal(got, call())
    del garbage


def _tensor(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _halve(t, *_):
    t.mul_(0.5)


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_points", [1, 40, 9261])
def test_one_frame(gpu_lib, precision, n_points):
    from pycpet_gb300 import esp_grid, field_grid

    x, q = (_tensor(a) for a in _charges(900, 1))
    p = _tensor(np.random.default_rng(2).uniform(-1.0, 1.0, (n_points, 3)))
    for clamp in (True, False):
        _record_and_replay(lambda: field_grid(p, x, q, precision=precision, clamp=clamp), (q,), _halve)
    _record_and_replay(lambda: esp_grid(p, x, q, precision=precision), (q,), _halve)


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_tables(gpu_lib, precision):
    from pycpet_gb300 import GridBatch, TopoBatch, topo_hist2d_sets

    rng = np.random.default_rng(3)
    frames = [(rng.uniform(-1.0, 1.0, (n, 3)), *_charges(200 + n, n)) for n in (1, 30, 700, 2000)]
    for kind in ("field", "esp"):
        gb = GridBatch(frames, kind=kind, precision=precision, device=True)
        _record_and_replay(gb.run, (gb.points,), _halve)
    lines = [{"x": x, "q": q, "starts": p[:200], "n_iter": 60, "step": 0.02, "half_dims": [1.5, 1.5, 1.5]}
             for p, x, q in frames]
    tb = TopoBatch(lines, precision=precision, device=True)
    _record_and_replay(tb.run, (tb.starts,), _halve)
    values = _tensor(rng.uniform(0.0, 4.0, (5000, 2)))
    off = [0, 700, 701, 701, 5000]
    _record_and_replay(lambda: topo_hist2d_sets(values, list(off), (20, 20), ((0.0, 5.0), (0.0, 5.0)), normalize=False),
                       (values,), _halve)  # (counts: an empty set divided by its total is NaN)


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("lines", [20, 700, 3000])
def test_streamlines_and_distances(gpu_lib, precision, lines):
    from pycpet_gb300 import chi2_distance_matrix, topo_lines

    x, q = (_tensor(a) for a in _charges(2500, 4))
    starts = _tensor(np.random.default_rng(5).uniform(-1.0, 1.0, (lines, 3)))
    caps = _tensor(np.full(lines, 50, np.int32))
    _record_and_replay(lambda: topo_lines(starts, caps, x, q, 0.02, [1.5] * 3, precision=precision), (starts,), _halve)
    h = _tensor(np.random.default_rng(6).random((lines % 90 + 2, 300)))
    _record_and_replay(lambda: chi2_distance_matrix(h, precision=precision), (h,), lambda t: t.pow_(2.0))
