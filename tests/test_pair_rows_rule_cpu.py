"""The rule that sends 257 .. 890 rows to the pair kernel with the weights on the M side, at shapes that were
timed on both sides: rows x N x K, and that kernel's time over the other one's (148 SMs)."""
import pytest

from vllm_gcu_b200.ops import cuda as C

TIMED = [
    # short K, tiles of 256 x 256 by pairs on the other side
    (610, 8192, 1024, 1.26), (445, 8192, 1024, 1.21), (800, 6144, 512, 1.17), (557, 32768, 256, 1.61),
    # one full wave of 128 x 128 tiles on the other side
    (384, 6200, 4096, 1.19), (369, 6152, 2048, 1.32), (607, 6152, 5120, 1.21), (361, 12040, 256, 1.58),
    # and where it pays
    (301, 6144, 4096, 0.79), (301, 28672, 4096, 0.78), (445, 36864, 7168, 0.84), (301, 7168, 2048, 0.83),
    (301, 6144, 512, 0.88), (544, 28672, 4096, 0.79), (576, 7168, 2048, 0.85), (667, 18432, 7168, 0.89),
    (800, 7168, 16384, 0.88), (850, 12288, 5120, 0.94), (420, 6200, 4096, 0.87), (800, 6200, 4096, 0.90),
]


@pytest.mark.parametrize("M,N,K,ratio", TIMED)
def test_the_faster_side_is_taken(M, N, K, ratio, monkeypatch):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    rows = C._pair_rows(M, N, K)
    assert bool(rows) == (ratio < 1)
    assert rows % 32 == 0 and 0 <= rows <= 256


@pytest.mark.parametrize("M", [256, 446, 500, 512, 700, 768, 891, 1000])
def test_full_tiles_and_few_weight_tiles_go_elsewhere(M, monkeypatch):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    assert not C._pair_rows(M, 28672, 4096) and not C._pair_rows(301, 24 * 256 - 256, 4096)


# us of tiles on pairs and of the kernel with 128-row tiles as measured: the rule takes the faster one
@pytest.mark.parametrize("M,N,K,pair,other", [
    (4096, 5120, 2048, 65.0, 85.4), (2945, 5120, 2048, 59.2, 78.8), (2433, 8192, 3072, 91.0, 111.1),
    (3862, 2560, 14336, 243.9, 304.9), (7098, 10240, 11264, 1108.1, 1280.3), (1025, 14336, 4096, 96.6, 117.9),
    (1375, 10240, 3072, 83.1, 80.1), (2118, 768, 4096, 29.5, 20.3), (1569, 3072, 256, 16.2, 13.1),
    (3248, 512, 14336, 72.5, 52.6), (1065, 1024, 1536, 14.0, 9.2)])
def test_pairs_or_tiles_of_128_rows(monkeypatch, M, N, K, pair, other):
    monkeypatch.setattr(C, "_sms", lambda: 148)
    C._pair_pays.cache_clear()
    assert C._pair_pays(M, N, K) == (pair < other)
    C._pair_pays.cache_clear()
