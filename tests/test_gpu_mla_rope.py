"""Fused latent cache update with 16-byte accesses and the kernel that takes every other layout, against 64 bits."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


def _rotate(x, cs, neox):
    R = x.shape[-1]
    c, s = cs[:, None, :R // 2], cs[:, None, R // 2:]
    u, v = (x[..., :R // 2], x[..., R // 2:]) if neox else (x[..., 0::2], x[..., 1::2])
    y = (u * c - v * s, v * c + u * s)
    return torch.cat(y, -1) if neox else torch.stack(y, -1).flatten(-2)


# widths that the 16-byte form takes, from its smallest, and others (R 8 and 24, L 20, an odd row pitch); one
# row, no heads, more heads than threads; in place and into a wider query; rows without a slot
@pytest.mark.parametrize("T,H,L,R,pitch", [(1, 1, 8, 16, 0), (3, 0, 512, 64, 8), (130, 128, 512, 64, 64),
                                           (5, 300, 256, 32, 0), (2, 3, 2048, 128, 8), (4, 3, 64, 8, 0),
                                           (4, 2, 64, 24, 8), (4, 3, 20, 16, 0), (3, 2, 64, 16, 1)])
@pytest.mark.parametrize("neox", [False, True])
@pytest.mark.parametrize("in_place", [False, True])
def test_against_64_bits(T, H, L, R, pitch, neox, in_place):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(T + L)
    q = torch.randn(T, max(H, 1), 2 * R, device="cuda", generator=g).to(torch.bfloat16)[..., R:] if H else None
    kv = torch.randn(T, L + R + pitch, device="cuda", generator=g).to(torch.bfloat16)[:, :L + R]
    w = (1 + 0.1 * torch.randn(L, device="cuda", generator=g)).to(torch.bfloat16)
    pos = torch.randint(0, 50, (T,), device="cuda", generator=g)
    a = torch.rand(50, R // 2, device="cuda", generator=g) * 6
    cs = torch.cat([a.cos(), a.sin()], 1)
    slots = torch.randperm(T + 16, device="cuda", generator=g)[:T]
    slots[T // 2] = -1 if T > 1 else slots[0]
    cache = torch.full((-(-(T + 16) // 16), 16, L + R), 7.0, dtype=torch.bfloat16, device="cuda")
    out = None if in_place or not H else torch.full((T, H, L + R), 7.0, dtype=torch.bfloat16, device="cuda")
    x = kv.double()
    latent = x[:, :L] * torch.rsqrt(x[:, :L].square().mean(-1, keepdim=True) + 1e-5) * w.double()
    pe = _rotate(x[:, None, L:], cs.double()[pos], neox)[:, 0]
    q_want = _rotate(q.double(), cs.double()[pos], neox) if H else None
    k_pe, kv_c = C.mla_rope_cache(q, kv, pos, cs, w, 1e-5, cache, slots, L, neox,
                                  q_out=None if out is None else out[..., L:], want_k_pe=True, want_kv_c=True)
    _native.check_status()

    def close(got, want):          # sums of 32 bits, one rounding to bf16
        assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())
    close(k_pe, pe)
    close(kv_c, latent)
    if H:
        close(q if out is None else out[..., L:], q_want)
    if out is not None:
        assert bool((out[..., :L] == 7.0).all())
    rows, used = cache.view(-1, L + R), slots >= 0
    close(rows[slots[used]], torch.cat([latent, pe], 1)[used])
    rest = torch.ones(len(rows), dtype=torch.bool, device="cuda")
    rest[slots[used]] = False
    assert bool((rows[rest] == 7.0).all())
