"""The look for meshes: strides found by search over x wherever they lie (below and
above one look's 257 intervals, at its bounds, longer than 16,384), and point sets
that mislead it, give the bits of the same points in another order; frames on both
sides of the limits on pairs and charges, alone and in one launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, nz):
    ax = [np.linspace(-0.02 * (n - 1), 0.02 * (n - 1), n) for n in (nx, ny, nz)]
    return np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)


def _charges(n):
    rng = np.random.default_rng(n)
    return rng.uniform(-9.0, 9.0, (n, 3)) + 15.0, rng.normal(0.0, 0.4, n)


@pytest.fixture
def no_refinement(gpu_lib):
    from pycpet_gb300 import set_field_refinement

    old = set_field_refinement(0.0)
    yield
    set_field_refinement(old)


def _same_as_shuffled(pts, n, precision):
    from pycpet_gb300 import esp_grid, field_grid

    x, q = _charges(n)
    order = np.random.default_rng(1).permutation(len(pts))
    for fn in (field_grid, esp_grid):
        np.testing.assert_array_equal(fn(pts, x, q, precision=precision)[order],
                                      fn(pts[order], x, q, precision=precision))


@pytest.mark.parametrize("precision,n", [("fp32c", 600), ("fp64", 40)])
@pytest.mark.parametrize("shape", [(40000, 1, 1), (9000, 4, 1), (200, 1, 256), (200, 1, 257), (200, 1, 258),
                                   (300, 2, 257), (8, 100, 100), (9, 130, 150), (4, 150, 150), (3, 150, 150),
                                   (7, 257, 257)])
def test_strides(no_refinement, shape, precision, n):
    _same_as_shuffled(_mesh(*shape), n, precision)


@pytest.mark.parametrize("precision,n", [("fp32c", 600), ("fp64", 40)])
def test_point_sets_that_mislead(no_refinement, precision, n):
    """x constant throughout, back to its first value later, changing one point early or
    late; y and z shifted in one plane."""
    base = _mesh(40, 30, 40)
    flat = base.copy()
    flat[:, 0] = 0.25
    back = base.copy()
    back[24000:25200, 0] = base[0, 0]
    early, late, shifted = base.copy(), base.copy(), base.copy()
    early[1199, 0] += 0.01
    late[1200, 0] = base[0, 0]
    shifted[6000:7200, 2] += 0.005
    for pts in (flat, back, early, late, shifted, np.concatenate([base, base])):
        _same_as_shuffled(pts, n, precision)


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_frames_with_and_without_a_look(no_refinement, precision):
    """Frames of few and many charges on meshes and on points in no order in one launch."""
    from pycpet_gb300 import GridBatch, esp_grid

    frames = []
    for i, n in enumerate((0, 15, 16, 511, 512, 3000, 20, 700, 5, 512)):
        x, q = _charges(n)
        pts = _mesh(21, 21, 21) if i % 3 else _mesh(11, 13, 17)
        frames.append((np.random.default_rng(i).permutation(pts) if i == 5 else pts, x, q))
    gb = GridBatch(frames, kind="esp", precision=precision)
    for (p, x, q), out in zip(frames, gb.split(gb.run())):
        order = np.random.default_rng(2).permutation(len(p))
        ref = esp_grid(p, x, q, precision=precision)
        np.testing.assert_array_equal(esp_grid(p[order], x, q, precision=precision), ref[order])
        tol = 1e-12 if precision == "fp64" else 2e-6   # other charge chunks than alone
        assert np.abs(out.reshape(-1) - ref).max() <= tol * max(np.abs(ref).max(), 1e-300)


@pytest.mark.parametrize("kind", ["field", "esp"])
@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_tables_of_small_frames(no_refinement, kind, precision):
    """Frames of one to nine tiles with room for columns in their last one and without,
    meshes and not: the bits of the same table with every frame's points shuffled."""
    from pycpet_gb300 import GridBatch

    shapes = [(8, 8, 8), (7, 8, 8), (5, 10, 10), (11, 11, 11), (12, 12, 14), (16, 16, 8), (16, 16, 16), (15, 15, 15), (6, 6, 6)]
    frames, shuffled, orders = [], [], []
    for i, s in enumerate(shapes * 3):
        pts = _mesh(*s)
        x, q = _charges((600, 900, 40)[i // len(shapes)])
        order = np.random.default_rng(i).permutation(len(pts))
        frames.append((pts, x, q))
        shuffled.append((pts[order], x, q))
        orders.append(order)
    a, b = (GridBatch(f, kind=kind, precision=precision) for f in (frames, shuffled))
    for order, u, v in zip(orders, a.split(a.run()), b.split(b.run())):
        np.testing.assert_array_equal(u[order], v)
