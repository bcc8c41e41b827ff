"""Launches whose CTAs run out of lines and hand their last ones over while other
warps of the CTA are between two steps: the same bits as the launch that hands
nothing over (the allocation-free entry point), many times over.  Frames of 12,800
charges, whose lines are handed over whatever their length; line counts around what a CTA holds (64 slots; 16 lines are handed over), step caps that make
slots run empty one by one, in groups and all at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("caps_of", ["spread", "groups", "equal"])
def test_handed_over_lines_keep_their_bits(gpu_lib, caps_of):
    import torch
    from pycpet_gb300 import _lib, topo_lines

    sms = gpu_lib.cpetgb_device_sms()
    rng = np.random.default_rng(8)
    n = 12800
    x = rng.uniform(-40.0, 40.0, (2 * n, 3))
    x = torch.from_numpy(x[np.linalg.norm(x, axis=1) > 3.0][:n].copy()).cuda()
    q = torch.from_numpy(rng.normal(0.0, 0.4, n)).cuda()
    half = np.array([1.5, 1.5, 1.2])
    for per_sm in (21, 40, 64, 65, 90):
        L = sms * per_sm + 3
        starts = torch.from_numpy(rng.uniform(-1.2, 1.2, (L, 3))).cuda()
        caps = {"spread": rng.integers(0, 300, L), "groups": 40 * rng.integers(1, 5, L), "equal": np.full(L, 60)}[caps_of]
        caps = torch.from_numpy(caps.astype(np.int32)).cuda()
        res = torch.empty((L, 2), dtype=torch.float64, device="cuda")
        steps = torch.empty(L, dtype=torch.int32, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        rc = gpu_lib.cpetgb_topo_lines_noalloc(_lib.FP32C, L, n, starts.data_ptr(), caps.data_ptr(), 0.01,
                                               half.ctypes.data, x.data_ptr(), q.data_ptr(), res.data_ptr(), None,
                                               steps.data_ptr(), stream)
        assert rc == 0, _lib.last_error()
        for _ in range(6):
            r, s = topo_lines(starts, caps, x, q, 0.01, half, precision="fp32c", return_steps=True)
            assert torch.equal(r, res) and torch.equal(s, steps)


def test_frames_beyond_the_records(gpu_lib):
    """A table of so many lines that its last frames have no hand-over records: their
    lines end where they started, with the bits of a launch of their own."""
    from pycpet_gb300 import TopoBatch, topo_lines

    per_frame = 16 * gpu_lib.cpetgb_device_sms() + 70
    n_frames = (1 << 18) // (16 * gpu_lib.cpetgb_device_sms()) + 4
    rng = np.random.default_rng(9)
    x = rng.uniform(-40.0, 40.0, (26000, 3))
    x = x[np.linalg.norm(x, axis=1) > 3.0]
    frames = []
    for f in range(n_frames):
        n = 12800 + f % 3
        frames.append({"x": x[:n], "q": rng.normal(0.0, 0.4, n), "starts": rng.uniform(-1.2, 1.2, (per_frame, 3)),
                       "n_iter": rng.integers(0, 12, per_frame).astype(np.int32), "step": 0.02,
                       "half_dims": [1.5, 1.5, 1.2]})
    res, steps = TopoBatch(frames, precision="fp32c").run(return_steps=True)
    for f in (0, 1, n_frames // 2, n_frames - 5, n_frames - 3, n_frames - 1):
        fr = frames[f]
        r, s = topo_lines(fr["starts"], fr["n_iter"], fr["x"], fr["q"], 0.02, [1.5, 1.5, 1.2], return_steps=True)
        at = slice(f * per_frame, (f + 1) * per_frame)
        np.testing.assert_array_equal(res[at], r)
        np.testing.assert_array_equal(steps[at], s)


# both sides of a Kahan run (2,048 sources) and of the work from which lines are handed
# over (7,680 charges when lines are long), with few and many lines per SM
@pytest.mark.parametrize("n,step,per_sm", [(2048, 0.01, 3), (2049, 0.01, 9), (2049, 0.01, 11), (4000, 0.01, 17),
                                           (7616, 0.0015, 22), (7680, 0.0015, 22), (7680, 0.02, 22)])
def test_routes_agree(gpu_lib, n, step, per_sm):
    """The launch as planned against the allocation-free one, a table of two such frames,
    and a table whose other frame's size puts it on the other route."""
    import torch
    from pycpet_gb300 import TopoBatch, _lib, topo_lines

    rng = np.random.default_rng(n)
    x = rng.uniform(-40.0, 40.0, (2 * n, 3))
    x = x[np.linalg.norm(x, axis=1) > 3.0][:n]
    q = rng.normal(0.0, 0.4, n)
    L = per_sm * gpu_lib.cpetgb_device_sms() - 5
    starts, caps = rng.uniform(-1.2, 1.2, (L, 3)), rng.integers(0, 150, L).astype(np.int32)
    half = np.array([1.5, 1.5, 1.2])
    want, want_steps = topo_lines(starts, caps, x, q, step, half, return_steps=True)
    dev = [torch.from_numpy(a).cuda() for a in (starts, caps, x, q)]
    res = torch.empty((L, 2), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rc = gpu_lib.cpetgb_topo_lines_noalloc(_lib.FP32C, L, n, dev[0].data_ptr(), dev[1].data_ptr(), step,
                                           half.ctypes.data, dev[2].data_ptr(), dev[3].data_ptr(), res.data_ptr(),
                                           None, None, stream)
    assert rc == 0, _lib.last_error()
    np.testing.assert_array_equal(res.cpu().numpy(), want)
    frame = {"x": x, "q": q, "starts": starts, "n_iter": caps, "step": step, "half_dims": half}
    other = dict(frame, x=x[: n // 3], q=q[: n // 3], starts=starts[:300], n_iter=caps[:300])
    for frames in ([frame, frame], [other, frame]):
        r, s = TopoBatch(frames, precision="fp32c").run(return_steps=True)
        np.testing.assert_array_equal(r[-L:], want)
        np.testing.assert_array_equal(s[-L:], want_steps)
