"""256 x 256 tiles on CTA pairs (gemm_pair.cu), called by itself: every epilogue, both tile shapes, ragged last row
tiles, one and several K blocks, launches that repeat their bits."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mt", ["1", "2"])
@pytest.mark.parametrize("M,N,K", [(1100, 512, 384), (2048, 1024, 4096), (1024, 256, 64), (8192, 768, 512),
                                   (256, 28672, 512), (200, 16384, 256), (600, 8192, 128), (1, 256, 64)])
def test_every_epilogue(M, N, K, mt, monkeypatch):
    from vllm_gcu_b200.ops import cuda as C
    monkeypatch.setenv("VLLM_B200_PAIR_MT", mt)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :K]
    w = torch.randn(N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    want = a.double() @ w.double().t()
    silu, gelu = torch.nn.functional.silu, torch.nn.functional.gelu
    p = want.view(M, N // 64, 2, 32)
    for epi, exact, slope in [(C.EPI_NONE, want, 1), (C.EPI_BIAS, want + bias.double(), 1),
                              (C.EPI_RELU2, want.clamp(min=0).square(), 12), (C.EPI_GELU, gelu(want), 2),
                              (C.EPI_SILU_MUL, (silu(p[:, :, 0]) * p[:, :, 1]).reshape(M, -1), 12),
                              (C.EPI_GELU_MUL, (gelu(p[:, :, 0], approximate="tanh") * p[:, :, 1]).reshape(M, -1), 12)]:
        first = None
        for _ in range(2):
            out = torch.full((M, exact.shape[1] + 8), 7.0, device="cuda", dtype=torch.bfloat16)
            rc = _native.lib().b200_gemm_pair(a.data_ptr(), a.stride(0), w.data_ptr(), K, out.data_ptr(), out.stride(0),
                                              M, N, K, bias.data_ptr(), epi, _native.stream_ptr())
            assert rc == 0, epi
            first = out if first is None else first
            assert torch.equal(out, first)
        # 32-bit sums in any order through the epilogue's slope, approximate exponentials (1e-6 of |x|), bf16
        err = (out[:, :exact.shape[1]].double() - exact).abs()
        assert bool((err <= 2.0 ** -8 * exact.abs() + slope * K * 2.0 ** -24 + 4e-5).all()), (epi, err.max())
        assert bool((out[:, exact.shape[1]:] == 7.0).all())
    _native.check_status()
