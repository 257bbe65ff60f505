"""The pair GEMM whose K blocks are shared by the pairs of a cluster (gemm_pair_slices.cu) at the edges of its tiles
and slices, against a 64-bit product."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    if torch.cuda.is_available():
        _native.check_status()


# rows around the multiples of 32 and of 256; weight tiles cut short in and behind the first CTA's half; K blocks of
# 64 cut short, as many as slices and a number that does not divide; more tiles than clusters run at once
@pytest.mark.parametrize("M,N,K", [(1, 8, 256), (32, 136, 264), (33, 256, 4160), (256, 200, 320), (257, 392, 520),
                                   (301, 4096, 1000), (640, 8192, 448)])
@pytest.mark.parametrize("rows", [32, 160, 256])
@pytest.mark.parametrize("slices", [2, 3, 4])
def test_every_epilogue(M, N, K, rows, slices):
    from vllm_gcu_b200.ops import cuda as C
    assert _native.lib().b200_gemm_pair_slices_at_once(slices) > 0
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :K]
    w = torch.randn(N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    want = a.double() @ w.double().t()
    silu, gelu = torch.nn.functional.silu, torch.nn.functional.gelu
    cases = [(C.EPI_NONE, want, 1), (C.EPI_BIAS, want + bias.double(), 1),
             (C.EPI_RELU2, want.clamp(min=0).square(), 12), (C.EPI_GELU, gelu(want), 2)]
    if N % 64 == 0:
        p = want.view(M, N // 64, 2, 32)
        cases += [(C.EPI_SILU_MUL, (silu(p[:, :, 0]) * p[:, :, 1]).reshape(M, -1), 12),
                  (C.EPI_GELU_MUL, (gelu(p[:, :, 0], approximate="tanh") * p[:, :, 1]).reshape(M, -1), 12)]
    for epi, exact, slope in cases:
        out = torch.full((M, exact.shape[1] + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        rc = _native.lib().b200_gemm_pair_slices(
            a.data_ptr(), a.stride(0), w.data_ptr(), K, out.data_ptr(), out.stride(0), M, N, K,
            bias.data_ptr(), epi, rows, slices, _native.stream_ptr())
        assert rc == 0
        got = out[:, :exact.shape[1]]
        # 32-bit sums in any order through the epilogue's slope, approximate exponentials (1e-6 of |x|), bf16
        err = (got.double() - exact).abs()
        assert bool((err <= 2.0 ** -8 * exact.abs() + slope * K * 2.0 ** -24 + 4e-5).all()), (epi, err.max())
        assert bool((out[:, exact.shape[1]:] == 7.0).all())


def test_refused():
    x = torch.zeros(64, 512, device="cuda", dtype=torch.bfloat16)
    args = (x.data_ptr(), 512, x.data_ptr(), 512, x.data_ptr(), 512, 64, 64)
    call = _native.lib().b200_gemm_pair_slices
    s = _native.stream_ptr()
    assert call(*args, 512, None, 0, 64, 5, s) == -20          # more pairs than a cluster has
    assert call(*args, 512, None, 0, 48, 2, s) == -20          # rows that are no multiple of 32
    assert call(*args, 512, None, 4, 64, 2, s) == -20          # fp32 results
    assert call(*args, 64, None, 0, 64, 2, s) == -20           # fewer K blocks than slices
    assert call(*args, 510, None, 0, 64, 2, s) == -2
    assert call(*args, 512, None, 1, 64, 2, s) == -5           # no bias


@pytest.mark.parametrize("M,N,K,head", [(160, 840, 520, 256), (301, 28672, 512, 28416), (257, 1088, 1000, 1024)])
def test_full_rounds_and_a_tail(M, N, K, head):
    """Two kernels in one call that meet at ``head``; nothing is written beside the result.  (Tolerance as above.)"""
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    exact = a.double() @ w.double().t()
    for epi in (C.EPI_BIAS, C.EPI_SILU_MUL) if N % 64 == 0 else (C.EPI_BIAS,):
        want = exact + bias.double()
        if epi == C.EPI_SILU_MUL:
            p = exact.view(M, N // 64, 2, 32)
            want = (torch.nn.functional.silu(p[:, :, 0]) * p[:, :, 1]).reshape(M, -1)
        out = torch.full((M, want.shape[1] + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        rc = _native.lib().b200_gemm_pair_rows_tail(
            a.data_ptr(), K, w.data_ptr(), K, out.data_ptr(), out.stride(0), M, N, K, bias.data_ptr(), epi, 160,
            head, 96, 2, _native.stream_ptr())
        assert rc == 0
        err = (out[:, :want.shape[1]].double() - want).abs()
        slope = 12 if epi == C.EPI_SILU_MUL else 1
        assert bool((err <= 2.0 ** -8 * want.abs() + slope * K * 2.0 ** -24 + 4e-5).all()), (epi, err.max())
        assert bool((out[:, want.shape[1]:] == 7.0).all())
