"""The cluster kernel of the smallest calls on a GPU that other streams keep busy, so
that the CTAs of a cluster do not all start at once: the bits are those of the tile
kernel, in which the same points are part of a larger frame (the charge chunks depend
on the number of 512-point tiles only)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["field", "esp"])
def test_clusters_that_start_with_skew(gpu_lib, kind):
    import torch
    from pycpet_gb300 import esp_grid, field_grid, set_field_refinement

    old = set_field_refinement(0.0)
    try:
        rng = np.random.default_rng(4)
        fn = esp_grid if kind == "esp" else field_grid
        pts = torch.from_numpy(rng.uniform(-1.0, 1.0, (300, 3))).cuda()
        load = torch.from_numpy(rng.uniform(-1.0, 1.0, (40000, 3))).cuda()
        frames = []
        for n in (8, 300, 2048, 8000, 32000):   # up to eight splits and beyond, a few charges per CTA and many
            x = torch.from_numpy(rng.uniform(-9.0, 9.0, (n, 3)) + 20.0).cuda()
            q = torch.from_numpy(rng.normal(0.0, 0.4, n)).cuda()
            frames.append((x, q, fn(pts, x, q)))
        streams = [torch.cuda.Stream() for _ in range(4)]
        torch.cuda.synchronize()
        got = []
        for i in range(120):
            x, q, more = frames[i % len(frames)]
            s = streams[i % 4]
            with torch.cuda.stream(s):
                if i % 3 == 0:
                    fn(load, frames[2][0], frames[2][1])
                k = 1 + i % 32
                got.append((k, fn(pts[:k], x, q), more))
        torch.cuda.synchronize()
        for k, few, more in got:
            assert torch.equal(few, more[:k])
    finally:
        set_field_refinement(old)
