"""Row sums of the prefill kernel of two heads: 32 keys each by themselves, so that small probabilities behind
a large one are not lost one by one."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


# the large probability in each chunk of 32 keys, as first and second of the two that are added first
@pytest.mark.parametrize("big", [0, 33, 64, 127])
def test_small_probabilities_behind_a_large_one(big):
    from vllm_gcu_b200.ops import cuda as C
    k = torch.zeros(8, 16, 1, 128, device="cuda", dtype=torch.bfloat16)
    flat = k.view(128, 128)
    flat[:, 0] = -24
    flat[big, 0] = 0
    q = torch.zeros(1, 2, 128, device="cuda", dtype=torch.bfloat16)
    q[..., 0] = 1
    cu = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    table = torch.arange(8, dtype=torch.int32, device="cuda")[None]
    # (probabilities are powers of two; more tiles than the step has bring it to this kernel)
    out, lse = C.varlen_prefill(q, k, torch.ones_like(k), table, cu, cu[1:] * 128, math.log(2), 300, return_lse=True,
                                num_q_tiles_128=150)
    _native.check_status()
    # of 127 times 2^-24 the one beside the large number may be lost, and a sum of the four chunks is rounded
    # thrice by 2^-24 at most; logarithm and scale 2^-24 of one
    want = math.log1p(127 * 2.0 ** -24)
    assert float((lse.double() - want).abs().max()) <= 5 * 2.0 ** -24, (lse - want) * 2 ** 24
    assert float((out - 1).abs().max()) <= 2.0 ** -8
