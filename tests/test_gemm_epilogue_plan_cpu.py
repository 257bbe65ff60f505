"""Dense GEMMs of more than 128 rows with GELU in the epilogue go to the kernel that is fast with it."""
import pytest

from vllm_gcu_b200.ops import cuda as C


# us of the kernel with the weights on the M side (its fastest tiles), of 256 x 256 tiles on pairs and of 128-row tiles,
# weights beyond L2
@pytest.mark.parametrize("M,N,K,epi,rows,pair,tiles", [
    (200, 12288, 1024, "GELU_MUL", 13.0, 12.0, 13.1), (200, 12288, 1024, "GELU", 16.1, 15.0, 15.4),
    (160, 8192, 2048, "GELU_MUL", 13.1, 15.9, 12.7), (160, 8192, 2048, "GELU", 15.3, 19.1, 14.8),
    (256, 16384, 2048, "GELU_MUL", 20.8, 18.1, 20.9), (256, 16384, 2048, "GELU", 24.7, 21.2, 26.3),
    (700, 11008, 1024, "GELU_MUL", 18.6, 16.5, 19.5), (700, 11008, 1024, "GELU", 26.7, 21.1, 28.5),
    (1500, 6144, 1024, "GELU_MUL", 18.9, 16.4, 18.9), (1500, 6144, 1024, "GELU", 26.4, 20.8, 28.6),
    (3000, 2048, 768, "GELU_MUL", 14.1, 12.8, 13.9), (3000, 2048, 768, "GELU", 19.7, 18.3, 20.9),
    (300, 6144, 4096, "GELU_MUL", 20.8, 27.0, 20.1), (300, 6144, 4096, "GELU", 22.9, 29.9, 22.5),
    (2048, 4096, 4096, "GELU_MUL", 48.4, 47.4, 52.5), (2048, 4096, 4096, "GELU", 53.1, 50.1, 61.8),
    (512, 16384, 512, "GELU_MUL", 16.3, 11.9, 13.2), (512, 16384, 512, "GELU", 23.7, 17.7, 24.7),
    (4096, 8192, 2048, "GELU_MUL", 86.5, 86.3, 100.5), (4096, 8192, 2048, "GELU", 96.6, 94.8, 132.0),
    (1000, 4096, 256, "GELU_MUL", 9.3, 7.3, 7.2), (1000, 4096, 256, "GELU", 13.1, 10.2, 13.0),
    (400, 8192, 1024, "GELU_MUL", 12.6, 11.3, 12.0), (400, 8192, 1024, "GELU", 16.5, 14.3, 16.8),
    (640, 6144, 2048, "GELU_MUL", 17.0, 16.8, 18.0), (640, 6144, 2048, "GELU", 21.0, 19.7, 23.5),
    (1200, 12288, 3072, "GELU_MUL", 65.1, 67.1, 82.0), (1200, 12288, 3072, "GELU", 69.0, 72.1, 98.6),
    (2500, 8192, 1024, "GELU_MUL", 35.9, 31.3, 39.9), (2500, 8192, 1024, "GELU", 52.6, 40.9, 62.3),
    (6000, 4096, 512, "GELU_MUL", 33.9, 24.1, 30.8), (6000, 4096, 512, "GELU", 54.9, 42.4, 58.9)])
def test_kernel_for_gelu(monkeypatch, M, N, K, epi, rows, pair, tiles):
    monkeypatch.setattr(C, "_SM_COUNT", 148)
    C._large_estimate.cache_clear()
    kind, _, slices = C._large_plan(M, N, K, False, getattr(C, "EPI_" + epi))
    C._large_estimate.cache_clear()
    took = {"rows": rows, "pair": pair, "tiles": tiles}[kind]
    assert slices == 1 and took <= 1.06 * min(rows, pair, tiles), kind
