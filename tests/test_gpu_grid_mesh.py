"""The grid kernels' special cases against their general path, bit for bit: a
mesh evaluated column by column and the same points in another order (which is
no mesh, so every point goes through the general loop), and frames of few points
against the same points inside a frame of more (same charge chunks: the chunks
depend on the number of 512-point tiles only)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, nz):
    ax = [np.linspace(-0.05 * (n - 1), 0.05 * (n - 1), n) for n in (nx, ny, nz)]
    return np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)


def _charges(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-9.0, 9.0, (n, 3)), rng.normal(0.0, 0.4, n)


def _both(kind, pts, x, q, precision, clamp):
    from pycpet_gb300 import esp_grid, field_grid

    if kind == "esp":
        return esp_grid(pts, x, q, precision=precision)
    return field_grid(pts, x, q, precision=precision, clamp=clamp)


@pytest.fixture
def no_refinement(gpu_lib):
    from pycpet_gb300 import set_field_refinement

    old = set_field_refinement(0.0)
    yield
    set_field_refinement(old)


FORMS = [("field", "fp32c", True), ("field", "fp32c", False), ("esp", "fp32c", True), ("field", "fp64", True),
         ("esp", "fp64", True)]


@pytest.mark.parametrize("kind,precision,clamp", FORMS)
@pytest.mark.parametrize("shape,n", [((4, 9, 9), 300), ((5, 11, 13), 1000), ((21, 21, 21), 700), ((11, 11, 11), 2500),
                                     ((7, 40, 1), 513), ((600, 1, 1), 257), ((3, 20, 20), 400), ((8, 1, 50), 1)])
def test_mesh_equals_shuffled_points(no_refinement, shape, n, kind, precision, clamp):
    pts = _mesh(*shape)
    x, q = _charges(n, n)
    x[0] = pts[len(pts) // 2]                       # one point on a charge: clamped tiles among the columns
    if not clamp or kind == "esp":
        x[0] += 0.3
    order = np.random.default_rng(1).permutation(len(pts))
    a = _both(kind, pts, x, q, precision, clamp)
    b = _both(kind, pts[order], x, q, precision, clamp)
    # (unclamped, a charge 0.3 A along the mesh lies on another point of it: the
    # same non-finite values in both)
    assert np.all(np.isfinite(a)) or not clamp or kind == "esp"
    np.testing.assert_array_equal(a[order], b)


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_almost_meshes(no_refinement, precision):
    """Truncated meshes, one moved point, a row off by the last bit of a double,
    signed zeros, repeated points: whatever is taken for a mesh, the values are
    those of the shuffled points."""
    x, q = _charges(900, 5)
    base = _mesh(9, 10, 11)
    cases = [base[:-1], base[:-37], base[1:], np.repeat(base[:1], 700, 0), np.concatenate([base, base])]
    moved = base.copy()
    moved[503, 2] += 1e-3
    last = base.copy()
    last[880:, 1] = np.nextafter(last[880:, 1], 9.0)
    zeros = base - base[len(base) // 2]
    zeros[::7] *= -1.0
    cases += [moved, last, zeros, base[:, [2, 1, 0]].copy(), base[::-1].copy()]
    for pts in cases:
        order = np.random.default_rng(2).permutation(len(pts))
        a = _both("field", pts, x, q, precision, True)
        np.testing.assert_array_equal(a[order], _both("field", pts[order], x, q, precision, True))


@pytest.mark.parametrize("kind,precision,clamp", FORMS)
@pytest.mark.parametrize("n", [0, 1, 31, 257, 8000, 33000])
def test_few_points_equal_more(no_refinement, n, kind, precision, clamp):
    """1 and 13 points (one cluster in FP32C up to 32,768 charges), 256 (one CTA per
    charge chunk) and 300 (the tile kernel)."""
    x, q = _charges(n, n + 3)
    x = x[:n] + 20.0 * (n > 0)
    pts = np.random.default_rng(3).uniform(-1.0, 1.0, (300, 3))
    if clamp and kind == "field" and n > 40:
        x[[3, 40]] = pts[[0, 12]]                   # on the charges: the clamp acts
    more = _both(kind, pts, x, q, precision, clamp)
    assert np.all(np.isfinite(more))
    for k in (1, 13, 256):
        few = _both(kind, pts[:k], x, q, precision, clamp)
        if precision == "fp32c":
            np.testing.assert_array_equal(few, more[:k])
        else:  # the FP64 runs and chunks of few points are shorter
            assert np.abs(few - more[:k]).max() <= 1e-13 * max(np.abs(more).max(), 1e-300)


def test_few_points_in_a_batch(no_refinement):
    """Frames of few and of many points, without points and without charges in
    one launch, more frames than a warp looks up at once."""
    from pycpet_gb300 import GridBatch

    frames = []
    for i in range(70):
        x, q = _charges((0, 5, 300, 1100)[i % 4], i)
        pts = (_mesh(6, 9, 7), np.random.default_rng(i).uniform(-1, 1, (i, 3)), _mesh(5, 5, 5)[: 3 * i])[i % 3]
        frames.append((pts, x + 15.0, q))
    for kind in ("field", "esp"):
        for precision in ("fp32c", "fp64"):
            gb = GridBatch(frames, kind=kind, precision=precision)
            for (p, x, q), out in zip(frames, gb.split(gb.run())):
                if len(p) == 0:
                    continue
                ref = _both(kind, p, x, q, precision, True).reshape(len(p), -1)
                tol = 1e-12 if precision == "fp64" else 2e-6
                assert np.abs(out - ref).max() <= tol * max(np.abs(ref).max(), 1e-300)
