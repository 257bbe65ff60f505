"""Decode attention gives the same bits wherever its splits merge, and steps keep their number of splits."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


def _step(lens, heads, kv_heads, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    count = [max(1, -(-n // 16)) for n in lens]
    table, at = torch.zeros(len(lens), max(count), dtype=torch.int32), 0
    for i, n in enumerate(count):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    kc, vc = (torch.randn(at, 16, kv_heads, 128, device="cuda", generator=g).to(dtype) for _ in range(2))
    q = torch.randn(len(lens), heads, 128, device="cuda", generator=g).to(dtype)
    return q, kc, vc, table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")


# few requests: the splits are a cluster; the same requests many times over: partial results in global memory
# and a second kernel.  1, 4 and 16 query heads per key head; splits and requests without keys; sinks and windows
@pytest.mark.parametrize("lens,heads,kv_heads,dtype,options", [
    ([640], 32, 8, torch.bfloat16, {}),
    ([1, 65, 0, 700], 8, 2, torch.bfloat16, {}),
    ([129, 500], 4, 4, torch.float16, {}),
    ([333, 1024], 32, 2, torch.bfloat16, {"sink": True}),
    ([900, 20], 16, 2, torch.bfloat16, {"window": 300}),
])
def test_merge_in_cluster_or_second_kernel(lens, heads, kv_heads, dtype, options):
    from vllm_gcu_b200.ops import cuda as C
    q, kc, vc, table, sl = _step(lens, heads, kv_heads, dtype)
    sink = torch.randn(heads, device="cuda") if options.get("sink") else None
    rest = dict(sink=sink, window=options.get("window", 0))
    times = -(-(2 * C._sms() + 1) // (2 * len(lens) * kv_heads))
    for splits in range(2, 9):
        assert len(lens) * kv_heads * splits <= 2 * C._sms() < times * len(lens) * kv_heads * splits
        few = C.paged_decode(q, kc, vc, table, sl, 128 ** -0.5, num_splits=splits, **rest)
        many = C.paged_decode(q.repeat(times, 1, 1), kc, vc, table.repeat(times, 1), sl.repeat(times),
                              128 ** -0.5, num_splits=splits, **rest)
        _native.check_status()
        assert torch.equal(few.repeat(times, 1, 1), many), splits


# (requests, key heads, keys): with another number of splits the probabilities are rounded otherwise
@pytest.mark.parametrize("B,kv_heads,most,want", [
    (1, 8, 640, 3), (12, 8, 900, 4), (64, 4, 2304, 2), (32, 8, 800, 2), (1, 8, 512, 1), (40, 8, 4000, 1),
    (1, 8, 16000, 32), (1, 1, 16000, 32)])
def test_steps_keep_their_number_of_splits(B, kv_heads, most, want):
    from vllm_gcu_b200.ops import cuda as C
    if C._sms() != 148:
        pytest.skip("stated for 148 SMs")
    lens = [most] + [1] * (B - 1)
    q, kc, vc, table, sl = _step(lens, 2 * kv_heads, kv_heads)
    assert C.decode_num_splits(B, kv_heads, most) == want
    got = C.paged_decode(q, kc, vc, table, sl, 128 ** -0.5, max_seq_len=most)
    assert torch.equal(got, C.paged_decode(q, kc, vc, table, sl, 128 ** -0.5, num_splits=want))
