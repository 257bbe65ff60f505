"""Prefill attention of two heads at once (attention_fmha_pair.cuh) at the edges of its tiles, windows and
rescaling, against attention in 64 bits; layouts around the rule that picks it.  Steps of fewer tiles of
single heads than SMs go to the kernel for one head; a tile count far above the step's, which is an upper
bound by contract, brings them to both."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    if torch.cuda.is_available():
        _native.check_status()


def _step(new, cached, kv_heads, block, gen, spread):
    """Keys and values in shuffled blocks, block table, offsets, lengths."""
    total = [n + c for n, c in zip(new, cached)]
    count = [-(-t // block) for t in total]
    caches = [torch.randn(sum(count) + 2, block, kv_heads, 128, device="cuda", generator=gen)
              for _ in range(2)]
    kc, vc = (caches[0] * spread).to(torch.bfloat16), caches[1].to(torch.bfloat16)
    order = torch.randperm(sum(count) + 2, generator=torch.Generator().manual_seed(1))
    table, at = torch.zeros(len(new), max(count), dtype=torch.int32), 0
    for i, n in enumerate(count):
        table[i, :n] = order[at:at + n]
        at += n
    cu = torch.tensor([0] + list(new)).cumsum(0).to(torch.int32).cuda()
    return kc, vc, table.cuda(), cu, torch.tensor(total, dtype=torch.int32, device="cuda")


# one token; rows and keys that end inside, at and just behind a tile of 128; cached prefixes; a step of
# several requests; windows inside a tile and across tiles; keys that are not masked; 2, 4, 6 and 8 heads
# per key head (pairs) and 1 and 3 (the kernel for one head); scores spread so far that the running
# maximum is raised in most tiles
@pytest.mark.parametrize("new,cached,heads,kv_heads,window,causal,block,spread", [
    ([1], [0], 2, 1, 0, True, 16, 1.0),
    ([128, 1, 127], [0, 128, 129], 4, 1, 0, True, 16, 1.0),
    ([5, 130, 64], [0, 0, 0], 8, 2, 0, True, 16, 1.0),
    ([129, 257], [1000, 15], 12, 2, 0, True, 32, 1.0),
    ([300], [63], 16, 2, 100, True, 16, 1.0),
    ([383], [5], 6, 1, 37, True, 16, 1.0),
    ([640], [700], 4, 2, 513, True, 16, 1.0),
    ([200], [56], 4, 2, 0, False, 16, 1.0),
    ([500, 40], [600, 0], 4, 2, 0, True, 16, 12.0),
    ([300], [0], 6, 2, 0, True, 16, 1.0),
    ([150], [20], 2, 2, 0, True, 16, 1.0),
])
def test_against_64_bits(new, cached, heads, kv_heads, window, causal, block, spread):
    from vllm_gcu_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(sum(new) + heads)
    kc, vc, table, cu, lens = _step(new, cached, kv_heads, block, gen, spread)
    wide = torch.randn(sum(new), heads * 128 + 64, device="cuda", generator=gen).to(torch.bfloat16)
    q = wide[:, :heads * 128].unflatten(1, (heads, 128))
    tiles = [sum(-(-n // t) for n in new) for t in (64, 128)]
    for extra in (0, 3, 150):                          # more tiles than the SMs of a B200
        out, lse = C.varlen_prefill(q, kc, vc, table, cu, lens, 128 ** -0.5, tiles[0] + extra,
                                    causal=causal, window=window, return_lse=True,
                                    num_q_tiles_128=tiles[1] + extra)
        for i, (n, c) in enumerate(zip(new, cached)):
            rows = slice(int(cu[i]), int(cu[i + 1]))
            used = table[i, :-(-(n + c) // block)].long()
            k, v = (x[used].flatten(0, 1)[:n + c].double().repeat_interleave(heads // kv_heads, 1)
                    for x in (kc, vc))
            s = torch.einsum("qhd,khd->hqk", q[rows].double(), k) * 128 ** -0.5
            pos = torch.arange(c, n + c, device="cuda")[:, None]
            key = torch.arange(n + c, device="cuda")[None]
            seen = key <= pos if causal else torch.ones(n, n + c, dtype=torch.bool, device="cuda")
            if window:
                seen = seen & (key > pos - window)
            s = s.masked_fill(~seen, float("-inf"))
            want = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v)
            # probabilities rounded to bf16 (2^-9 of the largest value), sums of 32 bits, scores to 2^-18 of
            # the largest, and the result rounded to bf16
            size = s.masked_fill(~seen, 0).abs().max()
            bound = (2.0 ** -9 + size * 2.0 ** -18) * v.abs().max() + 2.0 ** -8 * want.abs()
            assert bool(((out[rows].double() - want).abs() <= bound).all())
            assert (lse[:, rows].double() - torch.logsumexp(s, -1)).abs().max() <= 1e-5 + size * 2.0 ** -18


# one, two and six heads per key head: both kernels at the tile counts that the others above do not reach
@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 2), (6, 1)])
@pytest.mark.parametrize("window", [0, 70])
def test_sinks(heads, kv_heads, window):
    from vllm_gcu_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(heads)
    new, cached, block = [130, 1], [100, 64], 16
    kc, vc, table, cu, lens = _step(new, cached, kv_heads, block, gen, 1.0)
    q = torch.randn(sum(new), heads, 128, device="cuda", generator=gen).to(torch.bfloat16)
    sink = torch.randn(heads, device="cuda", generator=gen)
    for extra in (0, 150):
        out = C.fmha_prefill_sink(q, kc, vc, table, cu, lens, 128 ** -0.5, 3 + extra, sink, window=window)
        for i, (n, c) in enumerate(zip(new, cached)):
            rows = slice(int(cu[i]), int(cu[i + 1]))
            used = table[i, :-(-(n + c) // block)].long()
            k, v = (x[used].flatten(0, 1)[:n + c].double().repeat_interleave(heads // kv_heads, 1)
                    for x in (kc, vc))
            s = torch.einsum("qhd,khd->hqk", q[rows].double(), k) * 128 ** -0.5
            pos, key = torch.arange(c, n + c, device="cuda")[:, None], torch.arange(n + c, device="cuda")
            hidden = (key > pos) | (key <= pos - window if window else key < 0)
            s = s.masked_fill(hidden, float("-inf"))
            p = torch.softmax(torch.cat([s, sink.double()[:, None, None].expand(-1, n, 1)], -1), -1)
            want = torch.einsum("hqk,khd->qhd", p[..., :-1], v)
            bound = 2.0 ** -8 * (v.abs().max() + want.abs())
            assert bool(((out[rows].double() - want).abs() <= bound).all())
