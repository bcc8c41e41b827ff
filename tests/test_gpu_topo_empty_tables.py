"""A table of frames none of which has a line, with line offsets above zero: accepted
by a host call (which copies the whole extent back, rows of no frame undefined), a
device call and a replayed plan (which write nothing)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_offsets_without_lines(gpu_lib, precision):
    import torch
    from pycpet_gb300 import _lib

    prec = {"fp32c": _lib.FP32C, "fp64": _lib.FP64}[precision]
    desc = np.array([[0, 5, 3, 0], [5, 7, 1, 0]], np.int64)
    params = np.array([[0.01, 1.0, 1.0, 1.0]] * 2)
    starts, caps = np.zeros((3, 3)), np.full(3, 10, np.int32)
    x, q = np.random.default_rng(1).normal(0.0, 5.0, (12, 3)), np.ones(12)
    res, steps = np.full((3, 2), 7.0), np.full(3, 7, np.int32)
    args = [a.ctypes.data for a in (starts, caps, x, q, res)]
    assert gpu_lib.cpetgb_topo_batch(prec, _lib.HOST, 2, desc.ctypes.data, params.ctypes.data, *args, None,
                                     steps.ctypes.data, None) == 0, _lib.last_error()
    dev = [torch.from_numpy(a).cuda() for a in (starts, caps, x, q, np.full((3, 2), 7.0), np.full(3, 7, np.int32))]
    ptr = [t.data_ptr() for t in dev]
    stream = torch.cuda.current_stream().cuda_stream
    assert gpu_lib.cpetgb_topo_batch(prec, _lib.DEVICE, 2, desc.ctypes.data, params.ctypes.data, *ptr[:5], None,
                                     ptr[5], stream) == 0, _lib.last_error()
    plan = ctypes.c_void_p()
    assert gpu_lib.cpetgb_topo_plan_create(ctypes.byref(plan), prec, 2, desc.ctypes.data, params.ctypes.data,
                                           *ptr[:5], None, ptr[5]) == 0, _lib.last_error()
    assert gpu_lib.cpetgb_plan_launch(plan, stream) == 0, _lib.last_error()
    torch.cuda.synchronize()
    assert gpu_lib.cpetgb_plan_destroy(plan) == 0
    assert torch.all(dev[4] == 7.0) and torch.all(dev[5] == 7)
