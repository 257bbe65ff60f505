"""GEMMs of 129 rows and more add up K in one sum, whichever kernel the plan takes: the same bits as the 128-row
tiles give.  (Partial sums are as exact, but round otherwise, which layers of 16 bits carry on.)"""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


# few weight tiles, which a split of K would spread over more pairs, and a last round of a few tiles; weights on the M
# side, 256 x 256 tiles of pairs and 128-row tiles; odd row counts; gated and plain
@pytest.mark.parametrize("M,N,K,gated", [
    (150, 6144, 4096, False), (186, 4864, 14336, False), (200, 20480, 4096, True), (301, 4096, 14336, False),
    (301, 28672, 4096, True), (400, 5120, 2048, False), (520, 2048, 4096, False), (620, 6656, 8192, False),
    (1000, 2112, 7168, False), (1024, 4096, 4096, False), (2048, 2112, 1536, False)])
def test_same_bits_as_128_row_tiles(M, N, K, gated):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    epi = C.EPI_SILU_MUL if gated else C.EPI_NONE
    want = torch.empty(M, N // 2 if gated else N, device="cuda", dtype=torch.bfloat16)
    _native.call("b200_gemm_bf16", a.data_ptr(), K, w.data_ptr(), K, want.data_ptr(), want.stride(0), M, N, K,
                 None, None, 0, epi, _native.stream_ptr())
    assert torch.equal(C.gemm_bf16(a, w, epilogue=epi), want)
    _native.check_status()
