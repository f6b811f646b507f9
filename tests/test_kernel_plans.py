"""The host-side choices of tile widths and splits (no GPU): whatever they pick must be a launch the kernels take."""
import pytest

from marin_b200.kernels import ops


@pytest.mark.parametrize("T", [129, 300, 512, 1000, 1024, 2048, 3000, 4096, 8192])
@pytest.mark.parametrize("N,K", [(6144, 2560), (2560, 4096), (19456, 2560), (2560, 9728), (7168, 5120), (5120, 17408), (384, 1096), (1152, 64)])
def test_stream_k_is_planned_only_where_the_kernel_takes_it(T, N, K):
    bn = ops.stream_k_plan(T, N, K)
    assert ops.persistent_plan(T, N) in ops.PERSISTENT_TILES
    paired = ops.paired_plan(T, N, K)
    assert paired == ops.persistent_plan(T, N) or (-paired in ops.PERSISTENT_TILES and paired % 32 == 0)
    if bn is None:
        return
    assert bn in ops.STREAM_K_TILES
    across, rows = -(-T // bn), -(-N // 128)
    groups = ops.SM_COUNT // across
    assert across <= ops.SM_COUNT and rows >= groups          # a tile is shared by two CTAs at most
    assert bn <= 256                                          # the parked tiles fit the scratch (sized for 256)


def test_stream_k_can_be_switched_off(monkeypatch):
    assert ops.stream_k_plan(2048, 2560, 9728) == 256
    monkeypatch.setattr(ops, "stream_k", False)
    assert ops.stream_k_plan(2048, 2560, 9728) is None


@pytest.mark.parametrize("T,N,K", [(436, 5120, 17408), (600, 5120, 17408), (1000, 5120, 5120)])
def test_stream_k_follows_the_switch_of_pairs_whichever_was_asked_first(monkeypatch, T, N, K):
    plans = {}
    for first in (True, False):
        ops._stream_k_width.cache_clear()
        for pairs in (first, not first):
            monkeypatch.setattr(ops, "pair_tiles", pairs)
            plans[first, pairs] = ops.stream_k_plan(T, N, K)
    assert plans[True, True] == plans[False, True] and plans[True, False] == plans[False, False]


@pytest.mark.parametrize("T,N,K", [(1, 6144, 2560), (8, 2560, 9728), (16, 2560, 4096), (64, 151936, 2560), (128, 300, 200), (33, 1000, 72)])
def test_few_token_plan_keeps_every_slice_in_use(T, N, K):
    bn, splits = ops.gemm_plan(T, N, K)
    assert bn in (16, 32, 64, 128) and bn >= min(T, 128) and splits in (1, 2, 4, 8)
    nkb = -(-K // 64)
    per = -(-nkb // splits)
    assert (splits - 1) * per < nkb                            # no slice without k-blocks


@pytest.mark.parametrize("T", [129, 136, 200, 384, 700, 1184, 2048])
@pytest.mark.parametrize("N,K", [(1, 8), (128, 64), (1024, 3072), (2560, 9728), (3232, 2560), (4096, 1024), (6144, 4096), (19456, 2560)])
def test_plans_beyond_128_tokens_are_launches_the_kernels_take(T, N, K):
    """Slices of K that all have work, whole tiles instead only where there are fewer of them than SMs or many tokens say so anyway."""
    bn, splits = ops.gemm_plan(T, N, K)
    nkb = -(-K // 64)
    assert bn == 128 and splits in (1, 2, 4, 8) and (splits - 1) * -(-nkb // splits) < nkb
    tiles = -(-N // 128) * -(-T // 128)
    assert splits == 1 or (tiles < ops.SM_COUNT and -(-nkb // splits) >= 4)
    assert not ops.half_round(128, N, K) and not ops.many_tokens(128, N, True)


@pytest.mark.parametrize("T,N,K,widths", [(33, 48, 48, (16, 32)), (128, 64, 256, (16, 32)), (333, 512, 128, (16, 32)),       # 4.1 us for 5.7 by tiles of 48, 6.9 for 8.1, 5.7 for 6.7
                                          (333, 1024, 1024, (96,)), (333, 4096, 1024, (96,)), (333, 2560, 9728, (112,)), (16, 2560, 9728, (16,))])
def test_float32_tiles_where_they_were_measured_faster(T, N, K, widths):
    width, splits = ops.f32_plan(T, N, K)
    assert width in widths and splits in ((1, 4, 8) if N <= ops.F32_FEW_ROWS else (1, 2, 4))


@pytest.mark.parametrize("T,N,K,whole", [(256, 6144, 1024, True), (256, 6144, 4096, True), (512, 2560, 9728, True), (640, 2560, 4096, True),      # 9.0 us for 12.2 in slices, 20.4 for 22.1, 40.7, 20.5 for 22.2
                                         (256, 4096, 4096, False), (256, 2560, 2048, False), (129, 2560, 9728, False), (200, 1024, 3072, False)])  # 20.4 for 16.6 in four slices, ...
def test_whole_tiles_where_they_were_measured_faster(T, N, K, whole):
    assert ops.half_round(T, N, K) == whole and not ops.many_tokens(T, N)


@pytest.mark.parametrize("T,N,K", [(T, N, K) for T in (1, 16, 33, 128, 129, 256, 511, 700, 1200, 2048) for N in (8, 1024, 2560, 6144, 9000) for K in (8, 512, 2560, 9728)])
def test_parts_of_k_have_a_sum_each_in_every_plan(T, N, K):
    """As many parts as the slices and accumulators of the plan make, none without k-blocks, and in whole tiles no more than tensor memory has room for."""
    sums, (bn, splits), nkb = ops.sums_plan(T, N, K), ops.gemm_plan(T, N, K), -(-K // 64)
    assert sums in (1, 2, 4, 8) and (sums - 1) * -(-nkb // sums) < nkb and sums % splits == 0
    assert sums == splits or (T > 128 and sums == 2 * splits and bn == 128)
    if ops.half_round(T, N, K):
        for width in (ops.paired_plan(T, N, K), ops.persistent_plan(T, N)):
            assert ops._whole_tiles(width, T, N, K) == ((128, sums) if sums > 1 else (width, 1)) and sums <= 4


@pytest.mark.parametrize("E", [1, 8, 16, 32, 60, 128, 384, 512])
@pytest.mark.parametrize("h,ff,shared_ff", [(2560, 3648, 2432), (4096, 2048, 0), (2048, 768, 768), (256, 512, 1024)])
def test_parts_of_the_experts_last_products_cost_less_than_the_round_they_save(E, h, ff, shared_ff):
    """Whatever the experts' number and shares: no part is empty or short, what further parts write and read again is less than a round of weight tiles, and it
    fits the memory set aside for it."""
    for rows in (1, 2, 5, 12, 20, 33, 60, 96, 99, 150):                       # an expert's average share
        pairs = rows * E
        for shared_rows in ((0, pairs // 2 + 1) if shared_ff else (0,)):
            tile = ops._expert_tile(pairs, E, shared_rows)
            parts = ops._down_parts(min(pairs, E), pairs, shared_rows, tile, h, ff, shared_ff if shared_rows else 0)
            further = (parts - 1) * (pairs + shared_rows) * h * 4
            assert 2 * further <= ops.SM_COUNT * 128 * max(ff, shared_ff) * 2 and further <= ops.EXPERTS_PARTS_BYTES
            for k in (ff, shared_ff if shared_rows else 0):
                n = k // 64
                assert k == 0 or parts == 1 or (-(-n // parts) >= 8 and (parts - 1) * -(-n // parts) < n)


@pytest.mark.parametrize("H,K,dv", [(32, 8, 128), (16, 8, 32), (16, 4, 48)])
def test_mixed_weights_never_take_more_memory_than_the_heads_sums(H, K, dv):
    """Where a step's portions go to the kernels that mix the weights first, those fit what the heads' sums of as many tokens would take (the working memory's
    plan); few tokens for the keys they meet, and none that fills a tile of 16 queries, never go there."""
    for tokens in (16, 84, 200, 400, 512, 2048, 8192):
        for portions in (1, 2, 4, 19, 60):
            for blocks in (1, 6, 18, 35, 64, 200):
                longest = -(-tokens // portions)
                if not ops._pooled_mix_pays(tokens, portions, longest, blocks, K, dv):
                    continue
                assert longest >= 16
                tiles = sum(-(-n // 16) for n in [tokens // portions] * (portions - 1) + [tokens - tokens // portions * (portions - 1)])
                assert tiles <= ops._pooled_mix_tiles(tokens, portions)
                assert ops._pooled_mix_tiles(tokens, portions) * blocks * H * 16 * 32 * 2 <= tokens * H * K * dv * 4
    assert ops._pooled_mix_pays(2048, 1, 2048, 35, 8, 128) and not ops._pooled_mix_pays(2048, 1, 2048, 64, 8, 128)
    for blocks, few, many in ((2, 174, 175), (10, 103, 104), (19, 71, 72), (35, 45, 46)):
        assert not ops._pooled_mix_pays(few, 1, few, blocks, 8, 128) and ops._pooled_mix_pays(many, 1, many, blocks, 8, 128)
