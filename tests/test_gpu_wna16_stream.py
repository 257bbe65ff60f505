"""The de-quantising GEMM for few rows (gemm_wna16_stream.cu) at the edges of its tiles, packed tiles, K
slices and groups, against a 64-bit product with the stored weights."""
import pytest
import torch

from vllm_gcu_b200.ops import _native

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    if torch.cuda.is_available():
        _native.check_status()


# a single block of 64; packed tiles (256 columns of 4 bits, 128 of 8) that a row does not fill; ragged
# tiles of 128 weight rows; groups smaller than a block, and one group per row; one and several K slices;
# rows around the multiples of 16, at 128 (two CTAs per SM) and above
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K,g", [(128, 64, 32), (200, 320, 32), (130, 192, 64), (1000, 8192, 8192),
                                   (4096, 4160, 64), (6144, 4096, 128), (19072, 512, 128)])
def test_edges(bits, N, K, g):
    from vllm_gcu_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(bits + N + K)
    q = torch.randint(0, 1 << bits, (N, K), device="cuda", generator=gen).to(torch.uint8)
    qw = (q[:, 0::2] | (q[:, 1::2] << 4)).contiguous() if bits == 4 else q
    sc = (0.004 * (0.5 + torch.rand(N, K // g, device="cuda", generator=gen))).to(torch.bfloat16)
    zs = (torch.randint(0, 1 << bits, sc.shape, device="cuda", generator=gen) * sc.float()).to(sc.dtype)
    w = q.double() * sc.double().repeat_interleave(g, 1) - zs.double().repeat_interleave(g, 1)
    for M in (1, 16, 17, 33, 100, 128, 129, 256):
        wide = torch.randn(M, K + 8, device="cuda", generator=gen).to(torch.bfloat16)
        x = wide[:, :K]                                # rows with a pitch
        bias = torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16) if M % 2 else None
        got = C.gemm_wna16(x, qw, sc, zs, g, bits, bias)
        assert got is not None
        want = x.double() @ w.t()
        # every weight is rounded once to bf16 (8 bit: behind a multiply-add in 32 bits), the sums have 32
        # bits, the result is rounded to bf16
        bound = (2.0 ** -9 + K * 2.0 ** -24) * (x.double().abs() @ w.abs().t())
        if bias is not None:
            want = want + bias.double()
        err = (got.double() - want).abs()
        assert bool((err <= bound + 2.0 ** -8 * want.abs() + 1e-30).all()), (M, err.max())
        assert torch.equal(got, C.gemm_wna16(x, qw, sc, zs, g, bits, bias))


# groups of 128 whose scales come eight at a time: one such load a row, slices of K that begin inside of one (3 to 7
# packed tiles each), rows on both sides of the early start, scales off a 16-byte boundary and rows of
# scales that are no multiple of one (both go one by one)
@pytest.mark.parametrize("N,K,off", [(300, 1024, 0), (1000, 3072, 0), (4096, 14336, 0), (256, 11264, 0),
                                     (256, 2048, 4), (640, 2560, 0)])
def test_groups_of_128(N, K, off):
    from vllm_gcu_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    q = torch.randint(0, 16, (N, K), device="cuda", generator=gen).to(torch.uint8)
    qw = (q[:, 0::2] | (q[:, 1::2] << 4)).contiguous()
    G = K // 128
    buf = torch.zeros(2, N * G + 8, device="cuda", dtype=torch.bfloat16)
    sc, zs = (b[off:off + N * G].view(N, G) for b in buf)
    sc.copy_(0.004 * (0.5 + torch.rand(N, G, device="cuda", generator=gen)))
    zs.copy_(torch.randint(0, 16, (N, G), device="cuda", generator=gen) * sc.float())
    w = q.double() * sc.double().repeat_interleave(128, 1) - zs.double().repeat_interleave(128, 1)
    for M in (1, 33, 64, 65, 128, 200):
        x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
        got = C.gemm_wna16(x, qw, sc, zs, 128, 4)
        want = x.double() @ w.t()
        # as above
        bound = (2.0 ** -9 + K * 2.0 ** -24) * (x.double().abs() @ w.abs().t()) + 2.0 ** -8 * want.abs()
        assert bool(((got.double() - want).abs() <= bound + 1e-30).all()), M
        assert torch.equal(got, C.gemm_wna16(x, qw, sc, zs, 128, 4))
