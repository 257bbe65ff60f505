"""Experts with their choice held fixed: the kernels that stream the weights (gemm_stream.cu) and that pair
CTAs (gemm_pair_rows.cu) are no further from 64 bits than the row tiles of 128 (gemm_bf16.cu).  All of them
round where the others do: the rows behind the gate, the weighted rows of every expert, their sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,k,H,I,T", [(128, 8, 2048, 768, 64), (32, 8, 7168, 2048, 128),
                                       (16, 4, 1024, 512, 700)])
def test_error_against_64_bits(E, k, H, I, T, monkeypatch):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(E)
    x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    w13, w2 = (torch.randn(E, n, m, device="cuda", generator=g).mul_(m ** -0.5).to(torch.bfloat16)
               for n, m in ((2 * I, H), (H, I)))
    ids = torch.rand(T, E, device="cuda", generator=g).topk(k, -1).indices.to(torch.int32)
    probs = torch.rand(T, k, device="cuda", generator=g).softmax(-1)
    want = torch.zeros(T, H, device="cuda", dtype=torch.float64)
    for e in range(E):
        t, slot = (ids == e).nonzero(as_tuple=True)
        u = (x[t].double() @ w13[e].double().t()).view(-1, I // 32, 2, 32)
        h = (torch.nn.functional.silu(u[:, :, 0]) * u[:, :, 1]).reshape(-1, I)
        want.index_add_(0, t, (h @ w2[e].double().t()) * probs[t, slot].double()[:, None])

    def error(out):
        return float((out.double() - want).norm() / want.norm())
    grouped = C.gemm_bf16_grouped
    with monkeypatch.context() as m:
        m.setattr(C, "gemm_bf16_grouped", lambda *a, **kw: grouped(
            *a, **{n: v for n, v in kw.items() if n not in ("sorted_ids", "pairs", "tile_rows")}))
        base = error(C.fused_experts(x, w13, w2, probs, ids))
    assert base < 2.0 ** -7
    for rows in (0, 1 << 20):
        with monkeypatch.context() as m:
            m.setattr(C, "GROUPED_STREAM_ROWS", rows)
            # (results of another order of the sums round the other way here and there)
            assert error(C.fused_experts(x, w13, w2, probs, ids)) <= 1.01 * base
