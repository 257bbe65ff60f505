"""The GEMM that streams the weights past few rows (gemm_stream.cu) at the edges of its tiles, K slices
and of the rule that picks it, against a 64-bit product."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native, ref

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    if torch.cuda.is_available():
        _native.check_status()


# rows around the multiples of 16 and the two row tiles; widths with a ragged last tile of 128, fewer
# tiles than SMs (K split over 2 .. 8 CTAs) and more; K with a ragged last block of 64, K blocks that
# the slices do not share evenly, and fewer blocks than a split takes
SHAPES = [(1, 8, 8), (1, 4096, 4096), (3, 136, 72), (15, 200, 1000), (16, 128, 4160), (17, 640, 5120),
          (32, 6144, 4096), (31, 28672, 512), (32, 19072, 264), (33, 6144, 4096), (64, 2112, 7168),
          (65, 4096, 4160), (128, 8192, 4096), (129, 4096, 4104), (256, 2048, 4096), (250, 72, 14336),
          (32, 1024, 128), (27, 200, 512), (17, 8, 72)]       # K so short that rows go into more tiles


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_every_epilogue(M, N, K):
    from vllm_gcu_b200.ops import cuda as C
    assert C._stream_pays(M, N, K)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    wide = torch.randn(M, K + 8, device="cuda", generator=g).to(torch.bfloat16)
    a = wide[:, :K]                                    # rows with a pitch
    b = torch.randn(N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    want = a.double() @ b.double().t()
    # fp32 sums of K products in any order, |sum of |products|| about 0.8 for unit rows
    sums = K * 2.0 ** -24

    def close(got, exact, scale=1.0):
        half_step = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -23
        err = (got.double() - exact).abs()
        assert bool((err <= half_step * exact.abs() + scale * sums + 1e-30).all()), err.max()

    out = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    C.gemm_bf16(a, b, out=out[:, :N])
    close(out[:, :N], want)
    assert bool((out[:, N:] == 7.0).all())
    assert torch.equal(C.gemm_bf16(a, b), out[:, :N])      # the order of the sums is fixed
    close(C.gemm_bf16(a, b, epilogue=C.EPI_FP32), want)
    close(C.gemm_bf16(a, b, bias=bias), want + bias.double())
    # d relu2 = 2 |x| dx; the approximate exponentials of the gated forms are good to 1e-6 of |x|
    close(C.gemm_bf16(a, b, epilogue=C.EPI_RELU2), want.clamp(min=0).square(), 2 * 6)
    close(C.gemm_bf16(a, b, epilogue=C.EPI_GELU), torch.nn.functional.gelu(want), 2)
    if N % 64 == 0:
        parts = want.view(M, N // 64, 2, 32)
        for epi, act in ((C.EPI_SILU_MUL, torch.nn.functional.silu),
                         (C.EPI_GELU_MUL, lambda x: torch.nn.functional.gelu(x, approximate="tanh"))):
            exact = (act(parts[:, :, 0]) * parts[:, :, 1]).reshape(M, N // 2)
            close(C.gemm_bf16(a, b, epilogue=epi), exact, 2 * 6 + 6 * 6e-6 / sums)


def test_captured_in_a_graph():
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(5, 512, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(1024, 512, device="cuda", generator=g).to(torch.bfloat16)
    want = ref.gemm(x, w, out_dtype=torch.float32)
    out, side, graph = C.gemm_bf16(x, w), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        C.gemm_bf16(x, w, out=out)
    out.zero_()
    graph.replay()
    assert (out.float() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("kind,dtype", [(0, torch.float8_e4m3fn), (2, torch.int8)])
@pytest.mark.parametrize("N,K", [(8, 16), (136, 144), (640, 5120), (4096, 4112), (19072, 272)])
def test_eight_bit_operands(kind, dtype, N, K):
    """One-byte operands with a scale per row and per column; K blocks are 128 wide here."""
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(N + K)

    def operand(rows):
        if dtype == torch.int8:
            return torch.randint(-127, 128, (rows, K + 16), device="cuda", generator=g).to(dtype)[:, :K]
        return torch.randn(rows, K + 16, device="cuda", generator=g).to(dtype)[:, :K]
    w = operand(N)
    ws = torch.rand(N, device="cuda", generator=g) + 0.5
    for M in (1, 16, 33, 128, 129, 256):
        if not C._q8_stream_pays(M, N, K):
            continue
        x, xs = operand(M), torch.rand(M, device="cuda", generator=g) + 0.5
        bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16) if M % 2 else None
        got = C.gemm_q8(x, w, xs, ws, bias, kind)
        want = x.double() @ w.double().t() * xs.double()[:, None] * ws.double()
        # fp8 products are exact in 32 bits and summed there (int8: exactly); three roundings of the scaled
        # sum, then bf16
        size = (x.double().abs() @ w.double().abs().t()) * xs.double()[:, None] * ws.double()
        bound = 2.0 ** -8 * want.abs() + (K if kind == 0 else 4) * 2.0 ** -24 * size
        if bias is not None:
            want = want + bias.double()
            bound = bound + 2.0 ** -8 * bias.double().abs()
        assert bool(((got.double() - want).abs() <= bound + 1e-30).all()), M


@pytest.mark.parametrize("act", ["silu_mul", "relu2", "gelu", ""])
@pytest.mark.parametrize("E,N,K,counts", [
    (1, 64, 8, [1]), (4, 128, 72, [0, 1, 16, 17]), (5, 320, 264, [128, 0, 129, 300, 2]),
    (40, 192, 2048, [i % 7 for i in range(40)])])
def test_experts(E, N, K, counts, act, monkeypatch):
    """Rows sorted by expert in tiles of 128: experts without rows, tiles with 1 .. 128 rows in use, several
    tiles of one expert; the padding's rows stay as they were."""
    from vllm_gcu_b200.ops import cuda as C
    monkeypatch.setattr(C, "GROUPED_STREAM_ROWS", 1 << 20)
    g = torch.Generator(device="cuda").manual_seed(E + N)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[:, None]
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(1))].to(torch.int32).cuda()
    sid, eid, used, pos = C.moe_align(ids, E)
    pairs, pos = ids.numel(), pos.long()
    x = torch.randn(pairs, K, device="cuda", generator=g).to(torch.bfloat16)
    a = torch.full((sid.numel(), K), float("nan"), device="cuda", dtype=torch.bfloat16)
    a[pos] = x
    w = torch.randn(E, N, K, device="cuda", generator=g).div_(math.sqrt(K)).to(torch.bfloat16)
    scale = torch.rand(sid.numel(), device="cuda", generator=g) if act == "" else None
    gated = act == "silu_mul"
    out = torch.full((sid.numel(), N // 2 if gated else N), 7.0, device="cuda", dtype=torch.bfloat16)
    C.gemm_bf16_grouped(a, w, eid, used, silu_mul=gated, row_scale=scale, out=out,
                        act="" if gated else act, sorted_ids=sid, pairs=pairs)
    y = torch.einsum("pk,pnk->pn", x.double(), w[ids[:, 0].long()].double())
    if gated:
        parts = y.view(pairs, N // 64, 2, 32)
        want = (torch.nn.functional.silu(parts[:, :, 0]) * parts[:, :, 1]).reshape(pairs, N // 2)
    else:
        want = y.clamp(min=0).square() if act == "relu2" else torch.nn.functional.gelu(y) \
            if act == "gelu" else y * scale[pos].double()[:, None]
    err = (out[pos].double() - want).abs()
    assert bool((err <= 2.0 ** -8 * want.abs() + 12 * K * 2.0 ** -24 + 4e-5).all()), err.max()
    rest = torch.ones(sid.numel(), dtype=torch.bool, device="cuda")
    rest[pos] = False
    assert bool((out[rest] == 7.0).all())
