"""Prefill attention of two query tiles per CTA where a CTA goes through several pieces of work: order of the pieces
over more sequences than lanes, and the latent form over expanded keys, against attention in 64 bits."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    if torch.cuda.is_available():
        _native.check_status()


def _place(total, block, extra=2):
    count = [-(-t // block) for t in total]
    order = torch.randperm(sum(count) + extra, generator=torch.Generator().manual_seed(1))
    table, at = torch.zeros(len(total), max(count), dtype=torch.int32), 0
    for i, n in enumerate(count):
        table[i, :n] = order[at:at + n]
        at += n
    return table.cuda(), sum(count) + extra


def _want(q, k, v, cached, scale):
    """q [n, h, dk], k [m, h, dk], v [m, h, dv] in 64 bits, and the largest score."""
    s = torch.einsum("qhd,khd->hqk", q, k) * scale
    hidden = torch.ones(s.shape[1:], dtype=torch.bool, device="cuda").triu(cached + 1)
    p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
    return torch.einsum("hqk,khd->qhd", p, v), s.masked_fill(hidden, 0).abs().max()


# 40 sequences: more than a warp's lanes; lengths of several tiles beside one token, cached prefixes that are no
# multiple of a tile, more pieces than SMs (3 rounds of the grid)
@pytest.mark.parametrize("heads,kv_heads", [(8, 2), (24, 4)])
def test_many_sequences(heads, kv_heads):
    from vllm_gcu_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(heads)
    new = [1 + (i * 37) % 300 for i in range(40)]
    cached = [(i * 53) % 400 for i in range(40)]
    total = [a + b for a, b in zip(new, cached)]
    table, blocks = _place(total, 16)
    kc, vc = (torch.randn(blocks, 16, kv_heads, 128, device="cuda", generator=gen).to(torch.bfloat16)
              for _ in range(2))
    q = torch.randn(sum(new), heads, 128, device="cuda", generator=gen).to(torch.bfloat16)
    cu = torch.tensor([0] + new).cumsum(0).to(torch.int32).cuda()
    lens = torch.tensor(total, dtype=torch.int32, device="cuda")
    tiles = [sum(-(-n // t) for n in new) for t in (64, 128)]
    out = C.varlen_prefill(q, kc, vc, table, cu, lens, 128 ** -0.5, tiles[0], num_q_tiles_128=tiles[1])
    for i, (n, c) in enumerate(zip(new, cached)):
        rows = slice(int(cu[i]), int(cu[i + 1]))
        used = table[i, :-(-(n + c) // 16)].long()
        k, v = (x[used].flatten(0, 1)[:n + c].double().repeat_interleave(heads // kv_heads, 1) for x in (kc, vc))
        want, size = _want(q[rows].double(), k, v, c, 128 ** -0.5)
        # probabilities rounded to bf16 (2^-9 of the largest value), scores to 2^-18 of the largest, result to bf16
        bound = (2.0 ** -9 + size * 2.0 ** -18) * v.abs().max() + 2.0 ** -8 * want.abs()
        assert bool(((out[rows].double() - want).abs() <= bound).all())


# one token; rows that end in the first and in the second tile of a piece, at and behind their edges; keys that
# end inside, at and behind a tile; prefixes; more pieces than SMs; 40 sequences
@pytest.mark.parametrize("new,cached,heads,block", [
    ([1], [0], 3, 16),
    ([127, 128, 129], [0, 1, 127], 2, 16),
    ([255, 256, 257], [128, 0, 300], 3, 32),
    ([600], [1000], 8, 16),
    ([700, 130], [0, 63], 40, 16),
    ([1 + (i * 41) % 280 for i in range(40)], [(i * 59) % 300 for i in range(40)], 5, 16),
])
def test_latent_prefill(new, cached, heads, block):
    from vllm_gcu_b200.ops import cuda as C
    L, R = 512, 64
    gen = torch.Generator(device="cuda").manual_seed(sum(new) + heads)
    total = [a + b for a, b in zip(new, cached)]
    table, blocks = _place(total, block)
    cache = torch.randn(blocks, block, L + R, device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.randn(heads * 256, L, device="cuda", generator=gen) * L ** -0.5).to(torch.bfloat16)
    wide = torch.randn(sum(new) + 3, heads * 192 + 64, device="cuda", generator=gen).to(torch.bfloat16)
    q = wide[:, :heads * 192].unflatten(1, (heads, 192))
    cu = torch.tensor([0] + list(new)).cumsum(0).to(torch.int32).cuda()
    lens = torch.tensor(total, dtype=torch.int32, device="cuda")
    out = torch.full((sum(new) + 3, heads, 128), 7.0, dtype=torch.bfloat16, device="cuda")
    for extra in (0, 3):
        C.latent_prefill(q, cache, table, cu, lens, sum(-(-t // 128) * 128 for t in total) + 128 * extra,
                         sum(-(-n // 256) for n in new) + extra, w, 192 ** -0.5, out)
        for i, (n, c) in enumerate(zip(new, cached)):
            rows = slice(int(cu[i]), int(cu[i + 1]))
            used = table[i, :-(-(n + c) // block)].long()
            latent = cache[used].flatten(0, 1)[:n + c]
            kv = torch.einsum("ml,hdl->mhd", latent[:, :L].double(), w.double().view(heads, 256, L))
            k = torch.cat([kv[..., :128], latent[:, None, L:].double().expand(-1, heads, -1)], -1)
            want, size = _want(q[rows].double(), k, kv[..., 128:], c, 192 ** -0.5)
            # as above, with keys and values rounded to bf16 in front: 2^-9 of each of 128 products in a score
            # (|q| and |k| of it bounded by their norms), 2^-9 of a value
            err = 2.0 ** -9 * 192 ** -0.5 * (q[rows].double().norm(dim=-1).max() * kv[..., :128].norm(dim=-1).max())
            bound = (2.0 ** -8 + 2 * err + size * 2.0 ** -18) * kv[..., 128:].abs().max() + 2.0 ** -8 * want.abs()
            assert bool(((out[rows].double() - want).abs() <= bound).all())
            assert ((out[rows].double() - want).norm() / want.norm()) < 2.0 ** -7
        assert bool((out[sum(new):] == 7.0).all())


def test_refused():
    from vllm_gcu_b200.ops import cuda as C
    from vllm_gcu_b200.ops._native import NativeError
    q = torch.zeros(4, 2, 192, dtype=torch.bfloat16, device="cuda")
    cache = torch.zeros(2, 16, 576, dtype=torch.bfloat16, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    out = torch.zeros(4 * 2 * 128 + 4, dtype=torch.bfloat16, device="cuda")[4:].view(4, 2, 128)
    with pytest.raises(NativeError):         # rows of the output that do not start at 16 bytes
        C.latent_prefill(q, cache, torch.zeros(1, 1, **i32), torch.tensor([0, 4], **i32),
                         torch.tensor([4], **i32), 128, 1,
                         torch.zeros(512, 512, dtype=torch.bfloat16, device="cuda"), 1.0, out)
