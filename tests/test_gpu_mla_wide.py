"""Latent attention with two key tiles in flight, the first columns of a wide query in tensor memory
(attention_mla.cu): widths on both sides of the line, edges of key tiles and of row tiles, block sizes
that are no power of two, against a 64-bit reference."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,L", [(384, 384), (448, 64), (448, 448), (512, 256), (576, 320), (576, 512)])
@pytest.mark.parametrize("N,decode", [(128, True), (128, False), (33, True), (3, False)])
@pytest.mark.parametrize("bs", [16, 48])
def test_against_64_bits(W, L, N, decode, bs):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(W + L + N)
    seq = [1, 63, 64, 65, 129, 0, 200]
    new = [1] * len(seq) if decode else [1, 2, 64, 3, 43, 0, 7]
    B, mb = len(seq), -(-max(seq) // bs)
    cache = torch.randn(B * mb, bs, W, device="cuda", generator=g).to(torch.bfloat16)
    bt = torch.randperm(B * mb, device="cuda", generator=g).view(B, mb).to(torch.int32)
    sl = torch.tensor(seq, dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + list(torch.tensor(new).cumsum(0)), dtype=torch.int32, device="cuda")
    T = sum(new)
    q = torch.randn(T, N, W, device="cuda", generator=g).to(torch.bfloat16)
    scale, tq = W ** -0.5, 128 // N
    tiles = sum(-(-n // tq) for n in new)
    for splits in (1, 3):
        got = C.mla_attention(q, cache, bt, sl, None if decode else cu, tiles, max(seq), scale,
                              splits=splits, L=L)
        torch.cuda.synchronize()
        _native.check_status()
        t = 0
        for b, (s, n) in enumerate(zip(seq, new)):
            if n == 0 or s == 0:
                assert not got[t:t + n].any()
                t += n
                continue
            kv = cache[bt[b].long()].reshape(-1, W)[:s].double()
            sc = torch.einsum("qnw,sw->qns", q[t:t + n].double(), kv) * scale
            late = torch.arange(s, device="cuda")[None] > torch.arange(s - n, s, device="cuda")[:, None]
            p = sc.masked_fill(late[:, None], float("-inf")).softmax(-1)
            want = torch.einsum("qns,sl->qnl", p, kv[:, :L])
            # probabilities rounded to bf16 before the product, the result after it
            size = torch.einsum("qns,sl->qnl", p, kv[:, :L].abs())
            err = (got[t:t + n].double() - want).abs()
            assert bool((err <= 2.0 ** -8 * (size + want.abs()) + 1e-3).all()), (b, splits, err.max())
            t += n
