"""A launch that the runtime refuses is answered by the call that made it and by no later one."""
import ctypes

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


def test_refused_launch_is_answered_once():
    lib = _native.lib()
    t = ctypes.c_void_p(torch.zeros(256, device="cuda").data_ptr())
    # more heads than a grid has rows: refused by the runtime, nothing runs
    rc = lib.b200_decode_reduce(t, ctypes.c_longlong(128), t, t, 2, 1, 70000, 128, 0, None, 128,
                                ctypes.c_void_p(_native.stream_ptr()))
    assert rc > 0
    # a launch whose result comes from the runtime's last error
    ids = torch.zeros(4, device="cuda", dtype=torch.int64)
    prev = torch.arange(5, 9, device="cuda")
    index = torch.arange(4, device="cuda", dtype=torch.int32)
    from vllm_gcu_b200.ops import cuda as C
    C.feed_tokens(ids, prev, index, index, 4)
    torch.cuda.synchronize()
    assert ids.tolist() == [5, 6, 7, 8]
