"""Rotation of whole heads with the cache write, and with the norms of query and key heads in front
(cache.cu), against 64 bits; layouts around the rule that picks the kernel."""
import pytest
import torch

from vllm_gcu_b200.ops import _native, ref

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    if torch.cuda.is_available():
        _native.check_status()


def _want(x, D, pos, table, w, eps):
    """Norm and rotation of every head in 64 bits."""
    x = x.double().unflatten(1, (-1, D))
    if w is not None:
        x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()
    c, s = (t[:, None] for t in table.double()[pos].chunk(2, -1))
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1).flatten(1)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fp32_table", [False, True])
@pytest.mark.parametrize("norms", [False, True])
@pytest.mark.parametrize("T,Hq,Hkv,D", [(1, 1, 1, 64), (3, 7, 1, 128), (33, 32, 8, 128), (65, 5, 3, 64),
                                        (17, 4, 4, 256)])
def test_heads(T, Hq, Hkv, D, norms, fp32_table, dtype):
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(T + Hq + D)
    rows = torch.randn(T, (Hq + 2 * Hkv) * D + 8, device="cuda", generator=g).to(dtype)
    parts = [Hq * D, Hkv * D, Hkv * D, 8]
    q, k, v, rest = rows.split(parts, -1)
    q0, k0, v0, rest0 = (t.clone() for t in (q, k, v, rest))
    angle = torch.rand(50, D // 2, device="cuda", generator=g) * 6
    table = torch.cat([angle.cos(), angle.sin()], -1).to(torch.float32 if fp32_table else dtype)
    pos = torch.randint(0, 50, (T,), device="cuda", generator=g)
    slots = torch.randperm(16 * 8, device="cuda", generator=g)[:T]
    slots[T // 2] = -1                                  # a padding row: rotated, not cached
    kc, vc = (torch.full((8, 16, Hkv, D), 7.0, device="cuda", dtype=dtype) for _ in range(2))
    w = [(1 + 0.2 * torch.randn(D, device="cuda", generator=g)).to(dtype) for _ in range(2)]
    extra = dict(norms=(w[0], w[1], 1e-5)) if norms else {}
    assert C.rope_cache_flash(q, k, v, pos, table, True, D, slots, kc, vc, **extra)
    if not norms:
        w = [None, None]
    step = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12        # half a step of the result
    for got, was, weight in ((q, q0, w[0]), (k, k0, w[1])):
        want = _want(was, D, pos, table, weight, 1e-5)
        assert bool(((got.double() - want).abs() <= 2 * step * want.abs() + 1e-5).all())
    assert torch.equal(v, v0) and torch.equal(rest, rest0)
    live = slots >= 0
    for cache, src in ((kc, k), (vc, v)):
        flat = cache.view(-1, Hkv * D)
        assert torch.equal(flat[slots[live]], src[live])
        keep = torch.ones(len(flat), dtype=torch.bool, device="cuda")
        keep[slots[live]] = False
        assert bool((flat[keep] == 7.0).all())


@pytest.mark.parametrize("kv", [torch.float8_e4m3fn, torch.int8])
def test_eight_bit_cache(kv):
    """The bytes are those of the rotated rows, rounded to their type, over the scale."""
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(3)
    T, Hq, Hkv, D = 19, 4, 2, 128
    q, k, v = (torch.randn(T, h * D, device="cuda", generator=g).to(torch.bfloat16)
               for h in (Hq, Hkv, Hkv))
    table = torch.randn(T, D, device="cuda", generator=g)
    pos = slots = torch.arange(T, device="cuda")
    kc, vc = (torch.zeros(2, 16, Hkv, D, device="cuda").to(kv) for _ in range(2))
    ks, vs = (torch.tensor([s], device="cuda") for s in (0.031, 0.017))
    C.rope_cache_flash(q, k, v, pos, table, True, D, slots, kc, vc, ks, vs)
    for cache, src, s in ((kc, k, ks), (vc, v, vs)):
        f = src.float() * (1.0 / s)
        want = f.round().clamp(-128, 127).to(kv) if kv == torch.int8 else f.clamp(-448, 448).to(kv)
        assert torch.equal(cache.view(-1, Hkv * D)[:T].view(torch.uint8), want.view(torch.uint8))


def test_layouts_that_go_elsewhere():
    """Partial and neighbouring-pair rotation, head sizes outside of the kernel, rows off the 16-byte grid:
    as the torch formulation; norms are declined and nothing is written."""
    from vllm_gcu_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(5)
    for D, rot, neox, off in ((128, 64, True, 0), (128, 128, False, 0), (96, 96, True, 0),
                              (128, 128, True, 1)):
        T, Hq, Hkv = 9, 4, 2
        base = torch.randn(T, (Hq + 2 * Hkv) * D + 8, device="cuda", generator=g).to(torch.bfloat16)
        q, k, v = base[:, off:off + (Hq + 2 * Hkv) * D].split([Hq * D, Hkv * D, Hkv * D], -1)
        table = torch.randn(T, rot, device="cuda", generator=g)
        pos = torch.arange(T, device="cuda")
        w = torch.ones(D, device="cuda", dtype=torch.bfloat16)
        caches = [torch.zeros(1, 16, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        before = base.clone()
        assert not C.rope_cache_flash(q, k, v, pos, table, neox, D, pos, *caches, norms=(w, w, 1e-5))
        assert torch.equal(base, before) and not caches[0].any()
        if off:
            continue                       # (the general kernel moves cache rows in vectors of 16 bytes)
        want = ref.rotary_embedding(pos, q.contiguous(), k.contiguous(), D, table, neox)
        C.rope_cache_flash(q, k, v, pos, table, neox, D, pos, *caches)
        for got, exp in zip((q, k), want):
            assert (got.float() - exp.float()).abs().max() <= 2.0 ** -8 * exp.float().abs().max()
