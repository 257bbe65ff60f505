"""SiLU over every bf16 number: its division is one by an approximate reciprocal and a Newton step."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (factors of at most 1: the product of the largest gates stays finite)
@pytest.mark.parametrize("other", [1.0, -0.75])
def test_every_gate(other):
    from vllm_gcu_b200.ops import cuda as C
    gate = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(-1, 64)
    x = torch.cat([gate, torch.full_like(gate, other)], 1)
    got = C.activation(x, "silu").double()
    g = gate.double()
    want = torch.nn.functional.silu(g) * other
    # -inf times 0 is NaN in 32 bits, where exp(inf) divides; rounding to bf16, and a few ulps of the approximate
    # exponential of up to 88 (2^-21 of |x|); below 1e-35 the quotient may be zero
    bad = g.isnan() | (g == -float("inf"))
    assert bool(got[bad].isnan().all()) and not bool(got[~bad].isnan().any())
    inf = g == float("inf")
    assert bool((got[inf] == want[inf]).all())
    rest = ~bad & ~inf
    err = (got - want).abs()[rest]
    assert bool((err <= (2.0 ** -8 + 2.0 ** -20 * g[rest].abs()) * want[rest].abs() + 1e-35).all())
