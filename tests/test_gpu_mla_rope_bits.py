"""Fused latent cache update: rows that 16-byte accesses can take and rows that they cannot get the same bits."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,L,R", [(1, 2, 512, 64), (130, 16, 512, 64), (7, 3, 264, 32), (3, 1, 2048, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("neox", [False, True])
def test_same_bits_from_both_kernels(T, H, L, R, dtype, neox):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(T + L)
    kv = torch.randn(T, L + R, device="cuda", generator=g).to(dtype)
    q = torch.randn(T, H, R, device="cuda", generator=g).to(dtype)
    w = (1 + 0.1 * torch.randn(L, device="cuda", generator=g)).to(dtype)
    pos = torch.randint(0, 50, (T,), device="cuda", generator=g)
    a = torch.rand(50, R // 2, device="cuda", generator=g) * 6
    cs = torch.cat([a.cos(), a.sin()], 1)
    got = []
    for pitch in (8, 7):                       # rows from 16-byte boundaries, and not
        wide = torch.zeros(T, L + R + pitch, device="cuda", dtype=dtype)
        wide[:, :L + R] = kv
        cache = torch.zeros(-(-T // 16), 16, L + R, dtype=dtype, device="cuda")
        out = torch.zeros_like(q)
        k_pe, kv_c = C.mla_rope_cache(q, wide[:, :L + R], pos, cs, w, 1e-5, cache, torch.arange(T, device="cuda"), L, neox,
                                      q_out=out, want_k_pe=True, want_kv_c=True)
        _native.check_status()
        got.append((cache, out, k_pe, kv_c))
    for x, y in zip(*got):
        assert torch.equal(x, y)
