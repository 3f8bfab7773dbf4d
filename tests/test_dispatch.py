"""The decisions the kernels' dispatch takes from sizes alone (how a context is cut into ranges, which tile
shape a prompt portion's products get, whether they are cut along K), for a stated number of SMs: no GPU and
no library needed, so a change to a cost model shows here first.  The GPU tests measure nothing either; they
check the same rules on the device's own SM count and that every choice gives the right numbers."""

import pytest


@pytest.fixture(params=[148, 132, 80])
def ops_with_sms(request, monkeypatch):
    import sllm_b200.ops as ops
    cached = [getattr(ops, n) for n in dir(ops) if hasattr(getattr(ops, n), "cache_clear")]
    for f in cached:
        f.cache_clear()
    monkeypatch.setattr(ops, "num_sms", lambda: request.param)
    yield ops, request.param
    for f in cached:                   # nothing decided for this SM count outlives the test
        f.cache_clear()


def test_the_cut_of_a_context_fills_whole_waves(ops_with_sms):
    ops, sms = ops_with_sms
    slots = 2 * sms
    for requests in (1, 2, 3, 8, 12, 16, 20, 33, 48, 64, 100, 128):
        for nkv in (1, 2, 4, 8):
            for ctx in (1, 127, 128, 255, 256, 1000, 4096, 5000, 17000, 32768):
                s = ops.choose_splits(requests, nkv, ctx, 2)
                assert 1 <= s <= max(1, min(ops.MAX_SPLITS, ctx // ops.SPLIT_MIN_KEYS)), (requests, nkv, ctx, s)
                tiles = -(-(-(-ctx // s)) // 64)
                assert -(-ctx // (tiles * 64)) == s, (requests, nkv, ctx, s)          # no range without keys
                ctas = requests * nkv * s
                if s > 1 and ctas > slots:                                            # a second wave only if well filled
                    assert ctas / (-(-ctas // slots) * slots) > 0.6, (requests, nkv, ctx, s)
                # the mma.sync form's merge walks the ranges one by one: its cap holds
                assert ops.choose_splits(requests, nkv, ctx, 2, ops.MMA_MAX_SPLITS) <= ops.MMA_MAX_SPLITS
    if sms == 148:
        assert ops.choose_splits(8, 4, 4096, 2) in (8, 9)          # 256 or 288 CTAs for 296 places
        assert ops.choose_splits(16, 4, 4096, 2) == 4              # five ranges would be 320 CTAs: two waves
        assert ops.choose_splits(64, 4, 4096, 2) == 1
        assert ops.choose_splits(1, 4, 32768, 2) == 74             # 296 CTAs of seven key tiles
        assert ops.choose_splits(1, 4, 1024, 2) == 8               # ranges of two key tiles, not fewer
        for pairs, ctx in ((32, 256), (148, 256), (160, 768), (160, 1024), (196, 1024), (200, 2048), (220, 2048), (224, 4096), (232, 4096), (300, 512)):
            assert ops.choose_splits(pairs, 1, ctx, 2) == 1, (pairs, ctx)      # a wave or two of whole contexts: a cut and its merge do not pay
        assert ops.choose_splits(120, 1, 512, 2) == 2 and ops.choose_splits(32, 1, 512, 2) == 4


def test_the_cut_of_a_context_whose_ranges_a_cluster_merges(ops_with_sms, monkeypatch):
    """Ranges may be single key tiles where the cluster that merges them fits the GPU, and are what they were where it does not."""
    ops, sms = ops_with_sms
    places = {64: 3 * sms, 128: 2 * sms}
    monkeypatch.setattr(ops, "_tma_ctas_per_sm", lambda hd: places[hd] // sms)
    monkeypatch.setattr(ops, "tma_clustered", lambda tiles, nkv, s, hd: 2 <= s <= 8 and tiles * nkv * s * 100 <= places[hd] * (100 if s == 2 else 85))
    for requests in (1, 2, 4, 8, 16, 24, 48, 64, 128):
        for nkv in (1, 2, 4, 8):
            for ctx in (1, 64, 127, 128, 240, 256, 512, 1024, 4096, 12001, 32768):
                for hd in (64, 128):
                    s, old = ops.choose_tma_splits(requests, nkv, ctx, hd), ops.choose_splits(requests, nkv, ctx, ops._tma_ctas_per_sm(hd))
                    assert s == old or ops.tma_clustered(requests, nkv, s, hd) or s == 1, (requests, nkv, ctx, hd)
                    assert -(-ctx // (-(-(-(-ctx // s)) // 64) * 64)) == s, (requests, nkv, ctx, hd)          # no range without keys
    if sms == 148:
        for requests, nkv, ctx, hd, want in [(8, 4, 127, 128, 1), (8, 4, 256, 128, 4), (8, 1, 256, 128, 4), (4, 2, 256, 64, 4), (16, 2, 512, 128, 4), (8, 4, 540, 128, 5), (8, 4, 1024, 128, 6), (8, 4, 4096, 128, 8),
                                             (32, 2, 1024, 64, 4), (148, 1, 512, 128, 2), (149, 1, 512, 128, 1), (1, 4, 12001, 128, 63), (1, 4, 32768, 128, 74), (64, 4, 4096, 128, 1)]:
            assert ops.choose_tma_splits(requests, nkv, ctx, hd) == want, (requests, nkv, ctx, hd)


def test_products_of_17_to_32_tokens(ops_with_sms, monkeypatch):
    """Up to one tile an SM, from 12 Mi elements and from a K on; with a norm owed on the input the rotary epilogue takes short reductions."""
    ops, sms = ops_with_sms
    monkeypatch.setattr(ops, "linear_tc_takes", lambda M, N, K: True)
    pays = ops._tc_unsplit_pays
    assert [pays(M, 12288, 1024) for M in (16, 17, 32, 33)] == [False, sms >= 96, sms >= 96, False]
    wide = 128 * sms
    for N, K, plain, gated in [(6144, 2048, True, True), (6144, 2032, False, False), (wide, 1536, True, True), (wide + 1, 1536, False, False), (wide, 896, wide * 896 >= 12 << 20, False), (wide, 768, False, False)]:
        assert (pays(24, N, K), pays(24, N, K, True)) == (plain, gated), (N, K)
    assert ops._ws_rope32_ok(16 * 2 * sms, 1024) and not ops._ws_rope32_ok(16 * 2 * sms + 1, 1024) and not ops._ws_rope32_ok(1152, 1056)


def test_tile_shapes_of_a_prompt_portions_products(ops_with_sms):
    ops, sms = ops_with_sms
    pairs = sms // 2
    for M in (129, 256, 512, 1024, 2048, 4096, 8192):
        for N in (896, 1536, 2048, 3584, 4608, 5120, 8192, 18944, 37888):
            form = ops.pair_wide_cols(M, N)
            assert form in (False, True, 448, 384, 320)
            mt = -(-M // 256)
            if form is True:
                assert ops.pair_tiles_wide(M, N)
            if form not in (False, True):       # no more waves than the 512-wide tiles would take
                assert -(-(mt * -(-N // form)) // pairs) <= -(-(mt * -(-N // 512)) // pairs)
            if form is not False:               # wide tiles only where a pair has few tiles anyway
                assert -(-(mt * -(-N // 256)) // pairs) < 4
            if ops.pair_tiles_slim(M, N):
                assert 2 * mt * -(-N // 256) <= pairs
    if sms == 148:
        assert ops.pair_wide_cols(2048, 3584) == 448 and ops.pair_wide_cols(2048, 4608) is True
        assert ops.pair_wide_cols(1024, 5120) == 320 and ops.pair_wide_cols(4096, 1536) == 384
        assert ops.pair_wide_cols(2048, 18944) is False and ops.pair_wide_cols(2048, 5120) is False
        assert ops.pair_tiles_slim(512, 4608) and not ops.pair_tiles_slim(2048, 3584)


def test_slices_of_k_for_results_of_few_tiles(ops_with_sms):
    ops, sms = ops_with_sms
    for M in (129, 197, 256, 512, 768, 1024, 2048, 4096):
        for N, K in ((3584, 3584), (3584, 18944), (4608, 3584), (5120, 5120), (5120, 27648), (896, 4864), (8, 520)):
            s = ops.pair_splits(M, N, K)
            assert 1 <= s <= ops.PAIR_SPLIT_MAX
            if s > 1:                           # a slice keeps at least PAIR_SPLIT_MIN_BLOCKS k blocks
                assert -(-K // 64) // s >= ops.PAIR_SPLIT_MIN_BLOCKS
    if sms == 148:
        assert ops.pair_splits(197, 3584, 18944) > 1 and ops.pair_splits(512, 3584, 18944) > 1
        assert ops.pair_splits(2048, 3584, 18944) == 1 and ops.pair_splits(2048, 37888, 3584) == 1


class _Rows:
    """bfloat16 rows on a device, as far as a decision looks at them."""
    is_cuda = True

    def __init__(self, *shape):
        import torch
        self.shape, self.dtype = shape, torch.bfloat16


@pytest.fixture
def any_pair_product(ops_with_sms, monkeypatch):
    ops, sms = ops_with_sms
    monkeypatch.setattr(ops, "pair_supports", lambda M, N, K: K % 8 == 0)
    return ops, sms


def test_a_mixture_is_sorted_only_where_its_matrices_rows_suit_the_product(any_pair_product):
    """The grouped product reads the experts' columns of the down matrix, whose rows end with the shared expert's: whole 16-byte pieces."""
    ops, _ = any_pair_product
    sizes = dict(E=8, top=2, ff=4096, matrices=3)
    assert ops.moe_grouped_pays(_Rows(4096, 4096), **sizes)
    assert ops.moe_grouped_pays(_Rows(4096, 4096), **sizes, shared_ff=104)
    for shared in (100, 4, 1):
        assert not ops.moe_grouped_pays(_Rows(4096, 4096), **sizes, shared_ff=shared)
    assert not ops.moe_grouped_pays(_Rows(4096, 4096), 8, 2, 4096 + 32, 3) and not ops.moe_grouped_pays(_Rows(4096, 4096 + 32), 8, 2, 4096, 3)


def test_a_mixture_is_sorted_where_that_saves_more_than_it_costs(any_pair_product):
    """Up to 256 tokens every expert's product is one tile of rows in either form, so sorting saves nothing, however many experts there are; from some
    hundred tokens on it pays, the later the smaller the matrices.  Never where its buffers would be much the larger ones."""
    ops, _ = any_pair_product
    sizes = [(4096, 64, 2, 1408, 3), (4096, 8, 2, 14336, 3), (4096, 256, 8, 2048, 3), (2048, 8, 2, 1408, 2), (2048, 128, 8, 768, 3), (1024, 4, 1, 256, 3)]
    for W, E, top, ff, mats in sizes:
        for T in (1, 128, 129, 150, 200, 256):
            assert not ops.moe_grouped_pays(_Rows(T, W), E, top, ff, mats), (T, W, E)
        for T in (129, 300, 700, 2048, 8192, 32768):
            if ops.moe_grouped_pays(_Rows(T, W), E, top, ff, mats):
                assert ops.moe_grouped_bytes(T, W, E, top, ff, mats) <= max(256 << 20, 1.25 * T * E * ff * 2 * mats), (T, W, E)
    for T, W, E, top, ff, mats, shared, want in [(300, 2048, 64, 6, 1408, 3, 2816, True), (300, 4096, 8, 2, 14336, 3, 0, True), (512, 2048, 8, 2, 1408, 3, 2816, False),
                                                 (2048, 2048, 8, 2, 1408, 2, 2816, True), (1024, 2048, 8, 2, 1408, 2, 2816, False), (4096, 1024, 16, 4, 512, 2, 512, True),
                                                 (512, 1024, 16, 4, 512, 2, 512, False), (4096, 1024, 4, 1, 256, 3, 0, False), (2048, 4096, 8, 2, 2752, 3, 0, True),
                                                 (2048, 4096, 256, 8, 1024, 3, 0, True), (512, 4096, 256, 8, 1024, 3, 0, False)]:
        assert ops.moe_grouped_pays(_Rows(T, W), E, top, ff, mats, shared) == want, (T, W, E, ff)


def test_single_tokens_of_very_many_small_heads(ops_with_sms, monkeypatch):
    import torch
    ops, _ = ops_with_sms
    monkeypatch.setattr(ops, "_token_heads_fit", lambda dk, dv: True)

    class Step:
        num_seqs = 64
    for d, heads, removes, want in [(16, 16, True, True), (16, 17, True, False), (16, 64, False, True), (20, 64, True, True), (8, 64, True, False), (64, 64, True, True)]:
        state = torch.empty(1, heads, d, d)
        assert state.data_ptr() % 16 == 0
        assert ops.recurrence_token_supports(_Rows(64, 4096), state, Step, d, d, removes) == want, (d, heads, removes)


@pytest.mark.parametrize("most", [1, 2, 3, 5, 7, 100])
def test_chunks_of_long_portions_in_groups(most):
    """Every chunk is in one group, in order; a request's chunks go on where the group before stopped."""
    import sllm_b200.ops as ops
    counts = [10, 2, 1, 4, 1]
    seen = []
    for a, n, runs in ops.chunk_groups(counts, most):
        assert 1 <= n <= most and a == len(seen) and sum(c for _, _, c in runs) == n
        at = 0
        for r, first, c in runs:
            assert first == at and c >= 1
            seen += [r] * c
            at += c
    assert seen == [r for r, c in enumerate(counts) for _ in range(c)]


def test_portions_run_in_chunks_where_that_is_faster(monkeypatch):
    """Shapes measured in both forms, on both sides of the line (148 SMs): heads whose padding or very many short portions make the chunks the slower
    form, and long portions of which the walk is one chain."""
    import sllm_b200.ops as ops
    monkeypatch.setattr(ops, "num_sms", lambda: 148)

    class Step:
        def __init__(self, lens):
            self.q_lens, self.num_seqs = lens, len(lens)
    for kind, heads, dk, dv, lens, want in [
            ("gated64", 32, 64, 64, [2048], True), ("gated64", 32, 64, 64, [96], False), ("gated64", 64, 64, 64, [100] * 40, False), ("gated64", 32, 64, 64, [100] * 100, False),
            ("gated64", 8, 16, 16, [150] * 16, False), ("gated64", 32, 64, 64, [2048] + [1] * 7, True), ("gated64", 4, 32, 32, [1, 2, 3], False),
            ("gated128", 16, 128, 128, [2048], True), ("gated128", 16, 128, 128, [128], False), ("gated128", 16, 128, 128, [1000, 100, 100, 100], True),
            ("forget128", 16, 128, 128, [400] * 5, True), ("forget128", 16, 128, 128, [128], False), ("fixed64", 64, 64, 64, [1001, 700, 600], True), ("fixed64", 8, 16, 16, [96] * 100, False),
            ("delta64", 16, 64, 64, [512], True), ("delta64", 4, 32, 32, [96] * 100, False), ("delta128", 16, 128, 128, [2048], True),
            ("delta128", 32, 128, 128, [1000] * 8, True), ("delta128", 8, 128, 64, [96] * 100, False),
            ("general", 32, 64, 64, [2048], True), ("general", 32, 64, 64, [200] * 8, False), ("general", 4, 16, 16, [96] * 100, False), ("general", 8, 32, 32, [150] * 16, False)]:
        assert ops._chunks_pay(kind, Step(lens), 96, heads, dk, dv) == want, (kind, heads, dk, len(lens), lens[0])
