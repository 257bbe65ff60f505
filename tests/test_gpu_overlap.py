"""Kernels that start under the end of the one in front (common.cuh, launch_overlapped) give the bits that
they give one by one, with buffers that every round writes again."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


# rows of the weight-streaming, the 256-wide, the pair and the general GEMM
@pytest.mark.parametrize("rows", [1, 24, 96, 301, 1024])
def test_back_to_back_as_one_by_one(rows):
    from vllm_gcu_b200.ops import cuda as C
    H, I = 1024, 6144
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, H, device="cuda", generator=g).to(torch.bfloat16)
    up = torch.randn(I, H, device="cuda", generator=g).div_(math.sqrt(H)).to(torch.bfloat16)
    down = torch.randn(H, I, device="cuda", generator=g).div_(math.sqrt(I)).to(torch.bfloat16)

    def run(wait):
        y, h = x.clone(), torch.zeros(rows, I, device="cuda", dtype=torch.bfloat16)
        for _ in range(30):
            C.gemm_bf16(y, up, out=h)
            wait()
            C.gemm_bf16(h, down, out=y)
            wait()
        torch.cuda.synchronize()
        return y

    want = run(torch.cuda.synchronize)
    assert want.isfinite().all()
    for _ in range(3):
        assert torch.equal(run(lambda: None), want)
    _native.check_status()
