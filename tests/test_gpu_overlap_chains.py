"""Chains of kernels that start under the end of the ones in front give, issued at once and replayed from a
captured graph, the bits that they give when every call is waited for.  Buffers are written again by every
round, so that a kernel that reads or writes before its turn shows."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu
H, ROUNDS = 1024, 6


class _OneByOne:
    """The native library, every call waited for."""

    def __init__(self, lib):
        self._lib = lib

    def __getattr__(self, name):
        fn = getattr(self._lib, name)

        def call(*args):
            rc = fn(*args)
            torch.cuda.synchronize()
            return rc
        return call


def _compare(step, state, monkeypatch):
    """``step`` updates the tensors of ``state`` in place; rounds one by one, at once and from a graph."""
    start = [t.clone() for t in state]

    def run(go):
        for t, s in zip(state, start):
            t.copy_(s)
        torch.cuda.synchronize()
        go()
        torch.cuda.synchronize()
        return [t.clone() for t in state]

    def rounds():
        for _ in range(ROUNDS):
            step()
    rounds()                                            # workspaces and plans exist before the capture
    lib = _native.lib()
    with monkeypatch.context() as m:
        m.setattr(_native, "lib", lambda: _OneByOne(lib))
        want = run(rounds)
    assert all(bool(w.isfinite().all()) for w in want if w.is_floating_point())
    assert any(not torch.equal(w, s) for w, s in zip(want, start))
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        rounds()
    for go in (rounds, rounds, graph.replay, graph.replay):
        for got, w in zip(run(go), want):
            assert torch.equal(got, w)
    _native.check_status()


def _weights(gen):
    def make(n, k):
        return torch.randn(n, k, device="cuda", generator=gen).div_(math.sqrt(k)).to(torch.bfloat16)
    return make


# rows of the streaming GEMM, of its K = 1024 neighbours and of the pair GEMM; one and several key splits
@pytest.mark.parametrize("rows,splits", [(1, 4), (24, 1), (24, 3), (96, 2), (301, 2)])
@pytest.mark.parametrize("head_norms", [False, True])
def test_decode_layer(rows, splits, head_norms, monkeypatch):
    """norm, projection, rotation and cache write, attention over key splits and their merge, output
    projection, norm, gated projection, output projection, LM head, sampling."""
    from vllm_gcu_b200.ops import cuda as C
    heads, kv, D, I, bs, ctx, vocab = 8, 2, 128, 1536, 16, 200, 2048
    gen = torch.Generator(device="cuda").manual_seed(rows)
    w = _weights(gen)
    qkv_w, o_w, up_w, down_w, head_w = (w((heads + 2 * kv) * D, H), w(H, heads * D), w(2 * I, H),
                                        w(H, I), w(vocab, H))
    norms = [(1 + 0.1 * torch.randn(n, device="cuda", generator=gen)).to(torch.bfloat16)
             for n in (H, H, D, D)]
    per = -(-ctx // bs)
    caches = [torch.randn(rows * per, bs, kv, D, device="cuda", generator=gen).to(torch.bfloat16)
              for _ in range(2)]
    table = torch.arange(rows * per, device="cuda", dtype=torch.int32).view(rows, per)
    lens = torch.randint(1, ctx + 1, (rows,), device="cuda", generator=gen, dtype=torch.int32)
    pos = (lens - 1).long()
    slots = table[torch.arange(rows, device="cuda"), pos // bs].long() * bs + pos % bs
    angles = pos.new_ones(ctx, D // 2).float().cumsum(0) * 0.01
    rope = torch.cat([angles.cos(), angles.sin()], -1)
    embed = torch.randn(vocab, H, device="cuda", generator=gen).to(torch.bfloat16)
    x = torch.randn(rows, H, device="cuda", generator=gen).to(torch.bfloat16)
    res, ids = torch.zeros_like(x), torch.zeros(rows, device="cuda", dtype=torch.int64)
    qkv = torch.empty(rows, (heads + 2 * kv) * D, device="cuda", dtype=torch.bfloat16)
    att = torch.empty(rows, heads, D, device="cuda", dtype=torch.bfloat16)
    h = torch.empty(rows, I, device="cuda", dtype=torch.bfloat16)
    y, logits = torch.empty_like(x), torch.empty(rows, vocab, device="cuda", dtype=torch.bfloat16)
    ws = (torch.empty(rows * heads * splits * D, device="cuda"),
          torch.empty(rows * heads * splits, device="cuda"))

    def step():
        C.norm(x, norms[0], 1e-6, residual=res, out=y)
        C.gemm_bf16(y, qkv_w, out=qkv)
        q, k, v = qkv.split([heads * D, kv * D, kv * D], -1)
        assert C.rope_cache_flash(q, k, v, pos, rope, True, D, slots, *caches,
                                  norms=(norms[2], norms[3], 1e-6) if head_norms else None)
        C.paged_decode(q.unflatten(1, (heads, D)), *caches, table, lens, D ** -0.5, out=att,
                       num_splits=splits, workspace=ws, max_seq_len=ctx)
        C.gemm_bf16(att.flatten(1), o_w, out=y)
        C.norm(y, norms[1], 1e-6, residual=res, out=x)
        C.gemm_bf16(x, up_w, epilogue=C.EPI_SILU_MUL, out=h)
        C.gemm_bf16(h, down_w, out=x)
        C.gemm_bf16(x, head_w, out=logits)
        C.sample(logits, out=ids)
        x.add_(embed[ids])
    _compare(step, [x, res, ids, *caches], monkeypatch)


# experts with a few rows (weights streamed) and with many (CTA pairs)
@pytest.mark.parametrize("rows", [3, 40, 700])
def test_experts(rows, monkeypatch):
    """Router in 32 bits, choice, alignment, rows in place, two grouped products, weighted sum."""
    from vllm_gcu_b200.ops import cuda as C
    E, k, I = 16, 4, 256
    gen = torch.Generator(device="cuda").manual_seed(rows)
    gate = _weights(gen)(E, H)
    w13, w2 = (torch.randn(E, n, m, device="cuda", generator=gen).div_(math.sqrt(m)).to(torch.bfloat16)
               for n, m in ((2 * I, H), (H, I)))
    weight = torch.ones(H, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(rows, H, device="cuda", generator=gen).to(torch.bfloat16)
    res, scores = torch.zeros_like(x), torch.empty(rows, E, device="cuda")

    def step():
        y = C.norm(x, weight, 1e-6, residual=res)
        C.gemm_bf16(y, gate, out=scores, epilogue=C.EPI_FP32)
        probs, ids = C.moe_topk(scores, k, True)
        x.copy_(C.fused_experts(y, w13, w2, probs, ids))
    _compare(step, [x, res, scores], monkeypatch)


@pytest.mark.parametrize("rows", [2, 40, 200])
@pytest.mark.parametrize("kind", ["fp8", "int8", "wna4", "wna8"])
def test_quantised(rows, kind, monkeypatch):
    """Rows quantised by the norm and by themselves, 8-bit products, activation; packed weights."""
    from vllm_gcu_b200.ops import cuda as C
    I = 1536
    gen = torch.Generator(device="cuda").manual_seed(rows)
    weight = torch.ones(H, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(rows, H, device="cuda", generator=gen).to(torch.bfloat16)
    res = torch.zeros_like(x)
    if kind in ("fp8", "int8"):
        def make(n, m):
            q, s = C.per_token_quant(torch.randn(n, m, device="cuda", generator=gen).to(torch.bfloat16),
                                     kind)
            return q, s.flatten() / math.sqrt(m)

        def product(y, m):
            q, s = C.per_token_quant(y, kind)
            return C.gemm_q8(q, m[0], s, m[1], kind=0 if kind == "fp8" else 2)
    else:
        bits = int(kind[-1])

        def make(n, m):
            q = torch.randint(0, 256, (n, m * bits // 8), device="cuda", generator=gen)
            s = torch.full((n, m // 128), 2.0 ** (1 - bits) / math.sqrt(m), device="cuda")
            return q.to(torch.uint8), s.to(torch.bfloat16), (s * 2 ** (bits - 1)).to(torch.bfloat16)

        def product(y, m):
            return C.gemm_wna16(y, *m, 128, bits)
    up, down = make(2 * I, H), make(H, I)

    def step():
        y = C.norm(x, weight, 1e-6, residual=res)
        x.copy_(product(C.activation(product(y, up)), down))
    _compare(step, [x, res], monkeypatch)
