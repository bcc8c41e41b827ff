"""The field refinement's histogram over many points (shared-memory bins, several tiles
and frames per block) and over few: exactly the points whose |E|^2 lies below tau^2
times the frame's scale are refined, the scale being the lower edge of the bin (exponent
and 4 bits of the float |E|^2) that holds the lower median; all others keep their bits.
Points within 1e-6 of the threshold may fall on either side (numpy rounds |E|^2 without
fused multiply-adds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TAU = 0.15


def _cut(v):
    """Truncated to a float."""
    return (np.ascontiguousarray(v).view(np.int64) & ~np.int64(0x1FFFFFFF)).view(np.float64)


def _check(plain, refined):
    e = _cut(plain)
    m2 = (e * e).sum(1).astype(np.float32)
    ok = np.isfinite(m2)
    bins = m2[ok].view(np.uint32) >> 19
    scale = np.uint32(np.sort(bins)[(len(bins) - 1) // 2] << 19).view(np.float32)
    thr = np.float64(np.float32(TAU * TAU)) * np.float64(scale)
    low, high = m2 < thr * (1 - 1e-6), ~(m2 < thr * (1 + 1e-6))
    changed = (plain != refined).any(axis=1)
    np.testing.assert_array_equal(plain[high], refined[high])
    assert np.all(changed[low])
    return int(low.sum())


@pytest.fixture
def tau(gpu_lib):
    from pycpet_gb300 import set_field_refinement

    old = set_field_refinement(TAU)
    yield set_field_refinement
    set_field_refinement(old)


def _points(n, seed):
    return np.random.default_rng(seed).uniform(-3.0, 3.0, (n, 3))


def _charges(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-6.0, 6.0, (n, 3)), rng.normal(0.0, 0.4, n)


# one tile more or less than the limit of 300, a mesh, charges in one chunk and in several
@pytest.mark.parametrize("n_points", [299 * 512, 300 * 512 - 64 * 4, 300 * 512, 1000003])
@pytest.mark.parametrize("n_charges", [300, 2500])
def test_one_frame(tau, n_points, n_charges):
    from pycpet_gb300 import field_grid

    x, q = _charges(n_charges, 3)
    pts = _points(n_points, 1)
    refined = field_grid(pts, x, q)
    tau(0.0)
    assert _check(field_grid(pts, x, q), refined) > 0


@pytest.mark.parametrize("graph", [False, True])
def test_frames_of_many_sizes(tau, graph):
    import torch
    from pycpet_gb300 import GridBatch

    sizes = [1, 40000, 2, 33, 513, 3, 90000, 700, 5, 20000, 31, 1, 64000] * 2
    frames = [(_points(n, i), *_charges((40, 700, 3000, 9)[i % 4], i + 50)) for i, n in enumerate(sizes)]
    gb = GridBatch(frames, device=True, graph=graph)
    refined = [r.cpu().numpy() for r in gb.split(gb.run().clone())]
    again = [r.cpu().numpy() for r in gb.split(gb.run().clone())]
    tau(0.0)
    plain = GridBatch(frames, device=True, graph=graph)
    plain = [r.cpu().numpy() for r in plain.split(plain.run())]
    torch.cuda.synchronize()
    assert sum(_check(p, r) for p, r in zip(plain, refined) if len(p) > 2) > 100
    for a, b in zip(refined, again):
        np.testing.assert_array_equal(a, b)
