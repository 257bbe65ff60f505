"""Which requests of a latent-attention step have their keys and values expanded per head."""
from vllm_gcu_b200.ops import cuda as C

SIZES = (512, 128, 64, 128)        # latent, key, rotated and value columns


def test_runs_cover_the_requests_in_order():
    q = [1024, 3, 700, 2000, 2, 2, 300]
    s = [1024, 900, 900, 9000, 50, 2, 300]
    runs = C.latent_prefill_plan(q, s, 128, *SIZES)
    assert [a for a, _, _ in runs] == [0] + [b for _, b, _ in runs[:-1]] and runs[-1][1] == len(q)
    assert runs == [(0, 1, True), (1, 2, False), (2, 4, True), (4, 6, False), (6, 7, True)]


def test_workspace_is_bounded():
    limit = C.LATENT_PREFILL_BYTES // (128 * 512)
    runs = C.latent_prefill_plan([4000] * 9, [4000] * 9, 128, *SIZES)
    assert all(wide and (b - a) * 4096 <= limit for a, b, wide in runs) and len(runs) == 3
    assert C.latent_prefill_plan([4000], [limit + 1], 128, *SIZES) == [(0, 1, False)]


def test_other_sizes_and_short_requests_stay_absorbed():
    assert C.latent_prefill_plan([2000], [2000], 128, 512, 128, 64, 64) == [(0, 1, False)]
    assert C.latent_prefill_plan([2000], [2000], 16, 512, 64, 64, 64) == [(0, 1, False)]
    assert not any(w for _, _, w in C.latent_prefill_plan([2, 8, 63], [2, 8, 63], 128, *SIZES))
    assert not C.latent_prefill_plan([64], [1088], 128, *SIZES)[0][2]
    assert C.latent_prefill_plan([128], [1152], 128, *SIZES)[0][2]
    assert not C.latent_prefill_plan([128], [4224], 16, *SIZES)[0][2]
    assert not C.latent_prefill_plan([128], [100], 128, *SIZES)[0][2]      # lengths that do not belong together
    assert C.latent_prefill_plan([], [], 128, *SIZES) == []
