"""The gated activation that writes fp8 or int8 with a scale per row: the bytes of the activation followed by the
quantisation, for rows of one CTA and of clusters, kept in registers and computed again; and columns split over
CTAs: the bytes of a row do not depend on how many rows a call has."""
import pytest
import torch

from vllm_gcu_b200.ops import cuda as C

pytestmark = pytest.mark.gpu


def _x(T, width, dtype, pad=0):
    g = torch.Generator().manual_seed(T * 7 + width)
    x = (torch.randn(T, width + pad, generator=g) * 2).to(dtype).cuda()
    return x[:, :width]


@pytest.mark.parametrize("kind", ["fp8", "int8"])
@pytest.mark.parametrize("d", [8, 72, 264, 2048, 14336, 16392, 40000])
@pytest.mark.parametrize("T", [1, 3, 37, 64, 148, 149, 300])
def test_same_bytes_as_two_kernels(T, d, kind):
    for dtype, act, mode, pad in ((torch.bfloat16, "silu", "act_mul", 0), (torch.float16, "gelu", "act_mul", 16),
                                  (torch.bfloat16, "silu", "mul_act", 8), (torch.bfloat16, "identity", "plain", 0)):
        x = _x(T, d if mode == "plain" else 2 * d, dtype, pad)
        x[T // 2] = 0                                     # a row whose scale is the floor
        q, s = C.activation(x, act, mode, quant=kind + "_token")
        wq, ws = C.per_token_quant(C.activation(x, act, mode), kind)
        assert torch.equal(s, ws) and torch.equal(q.view(torch.uint8), wq.view(torch.uint8))


@pytest.mark.parametrize("T,valid", [(3, 2), (64, 40), (200, 0), (300, 150)])
def test_rows_in_use(T, valid):
    x = _x(T, 4096, torch.bfloat16)
    n = torch.tensor([valid], device="cuda", dtype=torch.int32)
    q = torch.full((T, 2048), 7, device="cuda", dtype=torch.uint8).view(C.FP8)
    got, s = C.activation(x, "silu", "act_mul", out=q, quant="fp8_token", valid_rows=n)
    wq, ws = C.per_token_quant(C.activation(x, "silu", "act_mul"), "fp8")
    assert torch.equal(got.view(torch.uint8)[:valid], wq.view(torch.uint8)[:valid])
    assert torch.equal(s[:valid], ws[:valid]) and (got.view(torch.uint8)[valid:] == 7).all()


@pytest.mark.parametrize("quant", [None, "fp8_group128", "fp8_static"])
@pytest.mark.parametrize("T,d", [(1, 14336), (5, 128), (12, 640), (64, 14336), (96, 1152), (200, 4224)])
def test_rows_do_not_depend_on_the_split(T, d, quant):
    x = _x(T, 2 * d, torch.bfloat16)
    kw = {"scale": torch.tensor([0.05], device="cuda")} if quant == "fp8_static" else {}
    many = C.activation(x.repeat(-(-600 // T), 1), "silu", "act_mul", quant=quant, **kw)   # one CTA a row
    few = C.activation(x, "silu", "act_mul", quant=quant, **kw)
    for a, b in zip(few if isinstance(few, tuple) else (few,), many if isinstance(many, tuple) else (many,)):
        assert torch.equal(a.contiguous().view(torch.uint8), b[:T].contiguous().view(torch.uint8))
