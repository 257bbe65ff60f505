"""The pair GEMM with the weights on the M side (gemm_pair_rows.cu) at the edges of its tiles, against a
64-bit product; the experts' form beside one and two row tiles of an expert."""
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


# rows around the multiples of 32 and of 256; weight tiles of 256 cut short, in and behind the first CTA's
# half; K blocks of 64 cut short; one tile and several rounds of all pairs
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (32, 136, 72), (33, 256, 4160), (256, 200, 512),
                                   (257, 392, 264), (301, 6144, 1000), (640, 28672, 128)])
@pytest.mark.parametrize("rows", [0, 32, 160])
def test_every_epilogue(M, N, K, rows):
    from vllm_gcu_b200.ops import cuda as C
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
        rc = _native.lib().b200_gemm_pair_rows(
            a.data_ptr(), a.stride(0), w.data_ptr(), K, out.data_ptr(), out.stride(0), M, N, K,
            bias.data_ptr(), epi, rows, _native.stream_ptr())
        assert rc == 0
        got = out[:, :exact.shape[1]]
        # 32-bit sums in any order through the epilogue's slope, approximate exponentials (1e-6 of |x|), bf16
        err = (got.double() - exact).abs()
        assert bool((err <= 2.0 ** -8 * exact.abs() + slope * K * 2.0 ** -24 + 4e-5).all()), (epi, err.max())
        assert bool((out[:, exact.shape[1]:] == 7.0).all())


def test_the_rule_takes_it():
    from vllm_gcu_b200.ops import cuda as C
    assert C._pair_rows(301, 6144) and C._pair_rows(384, 28672)
    assert not C._pair_rows(512, 28672) and not C._pair_rows(301, 4096)
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(301, 512, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(6144, 512, device="cuda", generator=g).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    got = C.gemm_bf16(x, w)
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-2).all())


@pytest.mark.parametrize("act", ["silu_mul", "relu2", "gelu", ""])
@pytest.mark.parametrize("E,N,K,counts", [
    (1, 64, 8, [1]), (4, 192, 72, [0, 129, 256, 17]), (3, 320, 264, [700, 0, 513]),
    (40, 256, 1024, [i * 11 % 270 for i in range(40)])])
def test_experts(E, N, K, counts, act, monkeypatch):
    from vllm_gcu_b200.ops import cuda as C
    monkeypatch.setattr(C, "GROUPED_STREAM_ROWS", 0)
    g = torch.Generator(device="cuda").manual_seed(E + N)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[:, None]
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(1))].to(torch.int32).cuda()
    cap = C.moe_align_cap(ids.numel(), E)
    rows = torch.empty(cap // 128, device="cuda", dtype=torch.int32)
    sid, eid, used, pos = C.moe_align(ids, E, cap, tile_rows=rows)
    assert torch.equal(rows.long(), (sid.view(-1, 128) < ids.numel()).sum(1))
    pairs, pos = ids.numel(), pos.long()
    x = torch.randn(pairs, K, device="cuda", generator=g).to(torch.bfloat16)
    a = torch.full((cap, K), float("nan"), device="cuda", dtype=torch.bfloat16)
    a[pos] = x
    w = torch.randn(E, N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    scale = torch.rand(cap, device="cuda", generator=g) if act == "" else None
    gated = act == "silu_mul"
    out = torch.full((cap, N // 2 if gated else N), 7.0, device="cuda", dtype=torch.bfloat16)
    C.gemm_bf16_grouped(a, w, eid, used, silu_mul=gated, row_scale=scale, out=out,
                        act="" if gated else act, sorted_ids=sid, pairs=pairs, tile_rows=rows)
    y = torch.empty(pairs, N, device="cuda", dtype=torch.float64)
    for e in range(E):
        mine = ids[:, 0] == e
        y[mine] = x[mine].double() @ w[e].double().t()
    if gated:
        p = y.view(pairs, N // 64, 2, 32)
        want = (torch.nn.functional.silu(p[:, :, 0]) * p[:, :, 1]).reshape(pairs, N // 2)
    else:
        want = y.clamp(min=0).square() if act == "relu2" else torch.nn.functional.gelu(y) \
            if act == "gelu" else y * scale[pos].double()[:, None]
    err = (out[pos].double() - want).abs()
    assert bool((err <= 2.0 ** -8 * want.abs() + 12 * K * 2.0 ** -24 + 4e-5).all()), err.max()
    rest = torch.ones(cap, dtype=torch.bool, device="cuda")
    rest[pos] = False
    assert bool((out[rest] == 7.0).all())
