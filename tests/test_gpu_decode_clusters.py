"""Decode attention whose splits are a cluster of CTAs that merge in shared memory, against attention in 64 bits."""
import math

import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


# every cluster size; splits without keys, requests without keys, one key, keys that end inside a tile of 64 and
# at its edge; 1, 3, 4, 8 and 16 query heads per key head (shares of a CTA that do not divide evenly); both
# 16-bit types; sinks, soft caps, windows and chunks
@pytest.mark.parametrize("lens,heads,kv_heads,dtype,options", [
    ([1, 64, 65, 0, 700], 8, 2, torch.bfloat16, {}),
    ([129, 500], 16, 16, torch.bfloat16, {}),
    ([1500], 6, 2, torch.float16, {}),
    ([333, 77, 1024], 32, 2, torch.bfloat16, {"sink": True}),
    ([900, 20], 16, 2, torch.bfloat16, {"window": 300}),
    ([900, 513], 8, 2, torch.bfloat16, {"chunk": 512, "sink": True}),
    ([640], 4, 1, torch.bfloat16, {"softcap": 20.0}),
])
def test_against_64_bits(lens, heads, kv_heads, dtype, options):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    count = [max(1, -(-n // 16)) for n in lens]
    table, at = torch.zeros(len(lens), max(count), dtype=torch.int32), 0
    order = torch.randperm(sum(count), generator=torch.Generator().manual_seed(1))
    for i, n in enumerate(count):
        table[i, :n] = order[at:at + n]
        at += n
    kc, vc = (torch.randn(sum(count), 16, kv_heads, 128, device="cuda", generator=g).to(dtype) for _ in range(2))
    q = torch.randn(len(lens), heads, 128, device="cuda", generator=g).to(dtype)
    sl, scale = torch.tensor(lens, dtype=torch.int32, device="cuda"), 128 ** -0.5
    sink = torch.randn(heads, device="cuda", generator=g) if options.get("sink") else None
    cap, window, chunk = options.get("softcap", 0.0), options.get("window", 0), options.get("chunk", 0)
    for splits in range(2, 9):
        out = C.paged_decode(q, kc, vc, table.cuda(), sl, scale, num_splits=splits, sink=sink, softcap=cap,
                             window=window, chunk=chunk)
        _native.check_status()
        for i, n in enumerate(lens):
            if n == 0:
                assert bool((out[i] == 0).all())
                continue
            lo = max(0, n - window) if window else (n - 1) // chunk * chunk if chunk else 0
            used = table[i, :count[i]].long()
            k, v = (x[used].flatten(0, 1)[lo:n].double().repeat_interleave(heads // kv_heads, 1) for x in (kc, vc))
            s = torch.einsum("hd,khd->hk", q[i].double(), k) * scale
            s = cap * torch.tanh(s / cap) if cap else s
            t = s if sink is None else torch.cat([s, sink.double()[:, None]], -1)
            want = torch.einsum("hk,khd->hd", torch.softmax(t, -1)[:, :n - lo], v)
            # probabilities and the result rounded to 8 bits (11 for fp16), scores and the cap to 2^-18
            step = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
            bound = (step + s.abs().max() * 2.0 ** -18) * v.abs().max() + step * want.abs()
            assert bool(((out[i].double() - want).abs() <= bound).all()), (splits, i)


@pytest.mark.parametrize("B,kv_heads,most,want", [
    (64, 4, 2304, 1), (32, 8, 800, 1), (20, 8, 4000, 1), (12, 8, 900, 2), (1, 8, 640, 5), (1, 8, 4000, 8),
    (1, 1, 100, 1), (1, 8, 1 << 17, 19), (1, 1, 1 << 20, 32)])
def test_number_of_splits(B, kv_heads, most, want):
    from vllm_gcu_b200.ops import cuda as C
    if C._sms() != 148:
        pytest.skip("stated for 148 SMs")
    assert C.decode_num_splits(B, kv_heads, most, True) == want
