"""The host-side choices of tile shapes and splits: pure functions of the sizes, checked on the CPU."""
import itertools

from llm_inference_lab_b200.kernels import ops


def test_decode_splits_fit_the_gpu_and_the_cluster():
    """Splits never ask for more CTAs than the SMs hold at once, never leave a CTA without keys,
    and the cluster path (2..8 splits) is only taken while all CTAs are resident together."""
    for n_decode, n_kv, group, kv, (keys, per_sm) in itertools.product(
            (1, 2, 8, 32, 64, 200), (1, 2, 4, 8), (1, 7, 16, 20), (1, 100, 640, 2048, 4096, 32768),
            ((128, 2), (192, 1))):
        s = ops.decode_splits(n_decode, n_kv, group, kv, keys, per_sm)
        ctas = n_decode * n_kv * (-(-group // 16))
        assert 1 <= s <= 32
        if s > 1:
            assert (s - 1) * keys < kv, "a split without keys"
            assert ctas * s <= per_sm * ops.sm_count(), "a second round of CTAs"


def test_decode_splits_short_contexts_are_not_split():
    assert ops.decode_splits(8, 2, 7, 100) == 1
    assert ops.decode_splits(1, 1, 1, 1) == 1


def test_decode_splits_benchmark_shapes():
    # batch 8 of the 0.5B shape at 640 keys: one round of the warps per CTA, merged in the cluster
    assert ops.decode_splits(8, 2, 7, 640) == 5
    # heads of 128 (12 warps x 16 keys per round, one CTA per SM), 32 requests: no room to split
    assert ops.decode_splits(32, 4, 7, 4096, 192, 1) == 1


def test_prefill_tiles_cover_the_cases_they_were_measured_on():
    pick = ops._pick_prefill_tiles
    # down projection of the 0.5B shape: one wave of 128-wide tiles, K split to fill it
    assert pick(2048, 896, 4864, True) == ("tc", 128, 1)
    assert pick(1024, 896, 4864, True) == ("tc", 128, 2)
    assert pick(512, 896, 4864, True) == ("tc", 128, 4)
    # the same product may not be split when its consumer cannot sum partial products
    assert pick(512, 896, 4864, False) == ("tc", 128, 1)
    # short K is never split
    assert pick(512, 896, 896, True) == ("tc", 128, 1)
    # long K and enough tiles for most pairs of SMs: the pair kernel
    assert pick(4096, 896, 4864, True)[0] == "pair"
    assert pick(2048, 3584, 18944, True)[0] == "pair"
    # beyond one wave the width with the cheaper waves
    assert pick(1024, 3584, 1536, True) == ("tc", 256, 1)


def test_prefill_tiles_are_always_a_shape_the_kernels_take():
    for T, n_out, K, partial in itertools.product((129, 256, 1000, 2048, 8192, 50000), (8, 896, 1152, 9728, 151936),
                                                  (64, 896, 4864, 18944), (False, True)):
        kind, bn, splits = ops._pick_prefill_tiles(T, n_out, K, partial)
        assert kind in ("tc", "pair") and bn in (128, 256) and splits >= 1
        if not partial or kind == "pair":
            assert splits == 1
        if splits > 1:
            assert -(-K // 64) // splits >= 16, "a split with too few k-tiles"
            assert -(-T // 128) * -(-n_out // bn) * splits <= ops.sm_count()


def test_delta_walk_shapes_are_what_the_kernel_takes():
    """Slices of whole warps of walkers, two columns a thread only where registers allow, narrow slices while every CTA
    finds an SM of its own, and no slice far beyond the state's columns."""
    for pairs, keys, vdim, q_len in itertools.product((1, 14, 56, 128, 2000), (1, 16, 64, 128, 129, 256), (1, 8, 24, 64, 128, 200),
                                                      (1, 2, 2048)):
        vs, cols = ops.delta_walk_shape(pairs, keys, vdim, q_len)
        assert cols in (1, 2) and vs % (8 * cols) == 0 and 0 < vs <= 32 * cols and vs < vdim + 8 * cols
        assert cols == 1 or keys <= 128
    assert ops.delta_walk_shape(14, 64, 64, 2048) == (16, 1) and ops.delta_walk_shape(56, 64, 64, 512) == (32, 1)
    assert ops.delta_walk_shape(128, 128, 128, 512) == (64, 2) and ops.delta_walk_shape(14, 64, 64, 1) == (32, 2)


def test_pair_splits_and_gated_tiles_cover_the_cases_they_were_measured_on():
    assert [ops._pair_splits(T, 3584, 18944) for T in (136, 300, 512, 700, 1024)] == [4, 2, 2, 1, 1]
    assert ops._pair_splits(1024, 1536, 8960) == 2 and ops._pair_splits(300, 1536, 8960) == 0
    assert ops._pair_splits(2048, 896, 4864) == 0 and ops._pair_splits(300, 896, 896) == 0
    for T, n_out, K in itertools.product((129, 256, 1000, 2048, 8192), (8, 896, 1152, 9728), (64, 896, 4864, 18944)):
        s = ops._pair_splits(T, n_out, K)
        assert s == 0 or -(-K // 64) // s >= 64 and -(-T // 256) * -(-n_out // 224) * s <= ops.sm_count() // 2
    assert ops._gated_on_pairs(2048, 4864) and ops._gated_on_pairs(300, 8960) and ops._gated_on_pairs(411, 4864)
    assert not ops._gated_on_pairs(300, 4864) and not ops._gated_on_pairs(300, 18944) and not ops._gated_on_pairs(130, 4864)


def test_segments_of_recurrences_cover_the_cases_they_were_measured_on():
    walk = ops.delta_walk_segments
    assert [walk(14, 64, 64, 2048), walk(28, 64, 64, 700), walk(56, 64, 64, 500), walk(112, 64, 64, 500)] == [6, 4, 1, 1]
    assert walk(12, 128, 128, 2048) == 4 and walk(14, 64, 64, 300) == 1 and walk(14, 256, 64, 2048) == 1
    assert ops.scan_segments(56, 2048) == 11 and ops.scan_segments(112, 700) == 5 and ops.scan_segments(448, 250) == 1
    assert ops.scan_segments(56, 319) == 1 and ops.scan_segments(1, 5000) == 32
    assert [ops.decay_scan_segments(*c) for c in ((12, 2048, 1), (8, 1000, 1), (64, 2048, 1), (80, 700, 2), (8, 460, 1), (42, 449, 1))] \
        == [12, 10, 2, 1, 4, 1]


def test_small_states_are_walked_in_segments_where_that_was_faster():
    """(channels, entries, requests, tokens) on either side of the line."""
    def cut(channels, N, requests, tokens):
        n = ops.scan_segments(requests * -(-channels // 32), tokens)
        return n > 1 and ops.scan_segments_pay(n, channels, N, requests, tokens)

    assert all(cut(*c) for c in ((64, 16, 1, 2048), (512, 16, 1, 2048), (512, 16, 1, 1000), (1024, 16, 1, 2048), (256, 16, 1, 8192),
                                 (512, 8, 1, 2048), (1792, 8, 1, 2048), (512, 4, 1, 330), (1792, 4, 1, 2048)))
    assert not any(cut(*c) for c in ((256, 16, 1, 319), (512, 16, 1, 330), (1024, 16, 1, 500), (1792, 16, 1, 2048), (1792, 16, 1, 700),
                                     (5120, 16, 1, 2048), (512, 16, 4, 500), (3072, 8, 1, 2048), (5120, 4, 1, 2048), (1792, 16, 64, 400)))


def test_rows_go_in_blocks_of_four_where_that_was_faster():
    """(rows of the longest portion, single rows beside it, head size)"""
    def pays(longest, singles, dim, portions=1):
        return ops.delta_rule_blocks(longest) and ops.delta_blocks_pay(longest, longest * portions + singles, portions + singles, dim)

    assert all(pays(*c) for c in ((64, 0, 64), (100, 8, 64), (500, 64, 64), (64, 0, 128), (400, 64, 128), (64, 0, 256), (500, 0, 32),
                                  (48, 0, 64, 8), (250, 0, 128, 7), (250, 0, 32, 8)))
    assert not any(pays(*c) for c in ((31, 0, 64), (48, 0, 64), (32, 64, 64), (100, 64, 64), (100, 64, 128), (200, 64, 128), (32, 0, 256),
                                      (100, 64, 256), (100, 0, 32)))


def test_decayed_recurrences_go_in_chunks_where_that_was_faster():
    """(heads, key channels, value columns, the requests' rows)"""
    def chunks(heads, keys, vdim, rows):
        return ops.decay_scan_chunks(len(rows) * heads * -(-vdim // 32), keys, max(rows), heads, vdim, sum(rows), len(rows))

    one = [1]
    assert all(chunks(*c) for c in ((14, 64, 68, [2048]), (14, 64, 68, [1000] * 2), (14, 64, 68, [250] * 8), (12, 128, 132, [1500]),
                                    (12, 128, 132, [300] * 4), (14, 64, 68, [500] + one * 32), (14, 64, 68, [2048] + one * 64),
                                    (14, 64, 68, [500] * 24), (4, 64, 64, [2048]), (32, 64, 64, [500] * 24)))
    assert not any(chunks(*c) for c in ((14, 64, 68, [449]), (14, 64, 68, [199] * 8), (14, 200, 68, [2048]), (14, 64, 68, [500] + one * 64),
                                        (12, 128, 132, [500] + one * 32), (32, 128, 128, [700] + one * 32), (64, 64, 64, [200] + [20] * 20)))
    # 16,384 rows of 64 heads of 128 x 128 would keep 1.1 GB of states
    assert not chunks(64, 128, 128, [16384]) and chunks(12, 128, 132, [16384])
    for heads, keys, vdim, rows in itertools.product((1, 14, 64), (16, 64, 128), (16, 132, 256), ([500], [450] + one * 200, [9000] * 8)):
        assert not chunks(heads, keys, vdim, rows) or 4 * (sum(rows) // 64 + len(rows)) * heads * keys * vdim <= ops.DECAY_SCAN_CHUNK_BYTES


def test_gated_products_take_the_kind_of_tile_whose_rounds_take_less_time():
    """By the measured costs of a round (pairs of SMs 0.9 of the small tiles' where K is long, the same where it is short),
    for every number of tokens."""
    for K, inter, cost in ((896, 4864, 1.0), (1536, 8960, 0.9), (3584, 18944, 0.9)):
        for T in range(129, 16385):
            pairs, small = -(-T // 256) * (inter // 128), -(-T // 128) * (inter // 128)
            if pairs >= 64:
                assert ops._gated_on_pairs(T, inter, K) == (cost * -(-pairs // 74) <= -(-small // 148)), (K, T)
    # seen to be faster on pairs, in one round more than the small tiles take
    assert all(ops._gated_on_pairs(T, 18944, 3584) for T in (1408, 1664, 2176, 2432, 4224))
    assert all(ops._gated_on_pairs(T, 8960, 1536) for T in (2432, 2944, 4224))
    assert not any(ops._gated_on_pairs(T, 4864, 896) for T in (300, 1408, 2432, 2944, 9856))
