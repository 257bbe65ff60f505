"""The rules that send rows to the pair kernel with the weights on the M side, at shapes that were
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


# us as measured with weights beyond L2, by kernel: tiles of 128, 160, 192, 224 and 256 rows with the weights on
# the M side, 256 x 256 tiles on pairs, 128-row tiles.  The plan's choice is within 12 per cent of the fastest.
@pytest.mark.parametrize("M,N,K,rows,pair,tiles", [
    (400, 5120, 2048, (18.8, 13.7, 13.7, 16.5, 16.5), 19.5, 19.3),
    (520, 4096, 14336, (95.4, 57.0, 61.3, 61.3, 60.3), 76.7, 91.0),
    (700, 28672, 4096, (148.1, 133.0, 128.3, 128.1, 121.7), 122.8, 145.6),
    (1024, 6144, 4096, (51.6, 51.9, 43.1, 48.3, 52.4), 53.7, 57.0),
    (1500, 4096, 14336, (174.1, 179.2, 143.1, 160.2, 181.8), 181.0, 182.8),
    (2048, 2112, 7168, (65.0, 63.7, 72.9, 83.7, 55.5), None, 69.1),
    (2048, 4096, 4096, (78.8, 63.7, 62.7, 70.3, 58.0), 57.1, 67.3),
    (2048, 32768, 512, (83.9, 80.5, 72.9, 80.0, 68.2), 81.6, 128.3),
])
def test_kernel_for_more_rows(monkeypatch, M, N, K, rows, pair, tiles):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    C._large_estimate.cache_clear()
    kind, r, _ = C._large_plan(M, N, K)
    C._large_estimate.cache_clear()
    took = {"pair": pair, "tiles": tiles}.get(kind) if kind != "rows" else None
    if kind == "rows":
        assert r % 32 == 0 and 32 <= r <= 256
        # (equal tiles: the smallest of the timed sizes that gives as many)
        same = [t for size, t in zip((128, 160, 192, 224, 256), rows) if -(-M // size) == -(-M // r)]
        took = min(same)
    assert took <= 1.12 * min(t for t in (*rows, pair, tiles) if t is not None)


def test_plans_cover_every_shape(monkeypatch):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    C._large_estimate.cache_clear()
    for M in (129, 257, 300, 1000, 5000, 100000):
        for N in (8, 264, 1000, 4096, 151936):
            for K in (8, 72, 512, 16384):
                kind, rows, slices = C._large_plan(M, N, K)
                assert kind in ("rows", "slices", "pair", "tiles") and rows % 32 == 0 and rows <= 256
                assert (2 <= slices <= 4 and K >= 512 * slices) if kind == "slices" else slices == 1
                assert kind != "pair" or N % 256 == 0 and K % 64 == 0
    C._large_estimate.cache_clear()


# us of the other kernels' best and with K split over the pairs of a cluster
@pytest.mark.parametrize("M,N,K,others,split", [
    (301, 4096, 14336, 49.9, 36.3), (301, 4096, 4096, 17.7, 15.2), (301, 2112, 7168, 24.8, 15.5),
    (400, 4096, 14336, 52.8, 44.0), (186, 4864, 14336, 50.0, 32.0), (175, 5632, 4096, 18.4, 14.8),
    (520, 2048, 4096, 17.3, 14.5), (256, 6144, 4096, 18.9, 20.3), (592, 2632, 1536, 9.3, 13.0),
    (740, 2816, 1024, 8.4, 12.9), (301, 6144, 4096, 19.5, 28.7), (400, 5120, 2048, 12.9, 21.5)])
def test_k_is_split_where_it_pays(monkeypatch, M, N, K, others, split):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    C._large_estimate.cache_clear()
    assert (C._large_plan(M, N, K)[0] == "slices") == (split < others)
    C._large_estimate.cache_clear()


# 129 .. 256 rows: us of the kernel with the weights on the M side over that of the kernel taken otherwise
@pytest.mark.parametrize("M,N,K,ratio", [
    (129, 28672, 4096, 0.90), (160, 10240, 2048, 0.73), (192, 28672, 4096, 0.93), (224, 36864, 7168, 0.96),
    (256, 10240, 2048, 0.81), (256, 9000, 3000, 0.80), (192, 7168, 1024, 0.80), (144, 16384, 512, 0.89),
    (256, 28672, 4096, 1.03), (256, 6144, 4096, 1.35)])
def test_weights_on_the_m_side_up_to_256_rows(monkeypatch, M, N, K, ratio):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    C._large_estimate.cache_clear()
    assert (C._large_plan(M, N, K)[0] == "rows") == (ratio < 1)
    C._large_estimate.cache_clear()


# us of one kernel, and of full rounds with a tail whose K is split
@pytest.mark.parametrize("M,N,K,one,tail", [
    (301, 28672, 4096, 74.5, 71.1), (400, 28672, 4096, 88.8, 83.6), (200, 20480, 4096, 48.7, 43.5),
    (310, 9728, 4096, 35.2, 30.8), (512, 10240, 5120, 49.3, 46.6),
    (300, 21504, 2048, 31.4, 34.3), (1000, 4864, 4096, 34.6, 36.2)])
def test_tail_where_it_pays(monkeypatch, M, N, K, one, tail):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    C._tail_plan.cache_clear(), C._large_estimate.cache_clear()
    plan = C._tail_plan(M, N, K)
    C._tail_plan.cache_clear(), C._large_estimate.cache_clear()
    assert (plan is not None) == (tail < one)
    if plan:
        assert plan[0] % 32 == 0 and plan[1] % 256 == 0 and 0 < plan[1] < N and 2 <= plan[3] <= 4
