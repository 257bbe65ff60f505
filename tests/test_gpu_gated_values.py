"""SiLU in the epilogues of the gated GEMMs gives what the activation kernel gives, which divides: the same bits
for every finite gate, those included whose 1 + exp(-x) is near the largest number."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


# rows of a call, each with gates of its own: weights streamed past few rows, weights on the M side, tiles
@pytest.mark.parametrize("rows", [1, 32, 128, 255, 2176])
@pytest.mark.parametrize("up", [1.0, -0.75])
def test_every_finite_gate(rows, up):
    from vllm_gcu_b200.ops import cuda as C
    from vllm_gcu_b200.ops import ref
    gate = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    gate = gate[gate.isfinite()]
    many, K = 256, 128
    gates = gate.view(-1, many)                    # [255, 256]
    # a row picks a set of 256 gates by a one, the weights hold the sets as columns
    for first in range(0, len(gates), K):
        w_gate = torch.zeros(many, K, device="cuda", dtype=torch.bfloat16)
        used = gates[first:first + K]
        w_gate[:, :len(used)] = used.t()
        w_up = torch.full((many, K), up, device="cuda", dtype=torch.bfloat16)
        w = ref.interleave_gate_up(w_gate, w_up)
        pick = torch.arange(rows, device="cuda") % len(used)
        a = torch.nn.functional.one_hot(pick, K).to(torch.bfloat16)
        got = C.gemm_bf16(a, w, epilogue=C.EPI_SILU_MUL)
        x = torch.cat([used[pick], torch.full((rows, many), up, device="cuda", dtype=torch.bfloat16)], 1)
        assert torch.equal(got, C.activation(x, "silu")), first
    _native.check_status()
