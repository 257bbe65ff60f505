"""Pairs sorted by expert, by one CTA and by clusters of them: around the numbers of pairs where the cluster grows and
where a thread has more pairs than it keeps in registers, with more experts than threads, experts that
are not local, tokens that do not count, and the weights of the sorted rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,E,mapped,valid", [
    (1, 1, 1, False, None), (1024, 1, 7, False, None), (1025, 1, 2048, False, None), (512, 4, 128, True, None),
    (513, 4, 3, False, 300), (1024, 4, 64, False, None), (1025, 4, 1500, True, 1000), (4096, 8, 128, False, None),
    (4100, 8, 128, True, 4097), (9000, 8, 384, False, None)])
def test_align(T, k, E, mapped, valid):
    from vllm_gcu_b200.ops import _native, cuda as C
    g = torch.Generator().manual_seed(T + E)
    n_all = 2 * E if mapped else E
    ids = torch.randint(0, n_all, (T, k), generator=g).to(torch.int32)
    ids[0, 0] = -1
    emap = None
    local = ids.clone()
    if mapped:
        emap = torch.full((n_all,), -1, dtype=torch.int32)
        emap[torch.randperm(n_all, generator=g)[:E]] = torch.arange(E, dtype=torch.int32)
        local = torch.where(ids >= 0, emap[ids.clamp(min=0).long()], -1)
    if valid is not None:
        local[valid:] = -1
    local = local.flatten().long()
    cap = C.moe_align_cap(T * k, E)
    rows = torch.full((cap // 128,), -7, dtype=torch.int32, device="cuda")
    w = torch.rand(T, k, generator=g).cuda()
    row_w = torch.full((cap,), -7.0, device="cuda")
    count = None if valid is None else torch.tensor([valid], dtype=torch.int32, device="cuda")
    sid, eid, used, pos = C.moe_align(ids.cuda(), E, cap, None if emap is None else emap.cuda(), count, rows, w, row_w)
    _native.check_status()
    n = torch.bincount(local[local >= 0], minlength=E)
    padded = (n + 127) // 128 * 128
    start = padded.cumsum(0) - padded
    total = int(padded.sum())
    assert int(used) == total
    experts = torch.repeat_interleave(torch.arange(E), padded // 128)
    eid, sid, pos = eid.cpu().long(), sid.cpu().long(), pos.cpu().long()
    assert torch.equal(eid[:len(experts)], experts) and bool((eid[len(experts):] == -1).all())
    tile = torch.arange(total // 128) * 128 - start[experts]
    assert torch.equal(rows.cpu().long()[:len(experts)], (n[experts] - tile).clamp(0, 128))
    assert bool((rows.cpu()[len(experts):] == 0).all())
    # every pair in a row of its expert, every row of an expert in use in front of its padding
    kept = local >= 0
    assert bool((pos[~kept] == -1).all())
    at = pos[kept] - start[local[kept]]
    assert bool(((at >= 0) & (at < n[local[kept]])).all())
    want = torch.full((cap,), T * k)
    want[pos[kept]] = kept.nonzero().flatten()
    assert torch.equal(sid, want) and int((sid < T * k).sum()) == int(kept.sum())
    weights = torch.cat([w.cpu().flatten(), torch.zeros(1)])
    assert torch.equal(row_w.cpu(), weights[want])


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (5, 3, 264), (300, 8, 2048), (3, 2, 7168)])
def test_scatter(T, k, H):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator().manual_seed(H)
    x = torch.randn(T, H + 8, generator=g).to(torch.bfloat16).cuda()[:, :H]
    pos = torch.randperm(T * k + 5, generator=g)[:T * k].to(torch.int32)
    pos[::3] = -1
    out = torch.full((T * k + 5, H), 7.0, dtype=torch.bfloat16, device="cuda")
    C.call("b200_moe_scatter", C.ptr(x), x.stride(0), C.ptr(out), H, C.ptr(pos.cuda()), T, k, H, 0, C.stream_ptr())
    want = torch.full((T * k + 5, H), 7.0, dtype=torch.bfloat16)
    keep = pos >= 0
    want[pos[keep].long()] = x.cpu()[keep.nonzero().flatten() // k]
    assert torch.equal(out.cpu(), want)
