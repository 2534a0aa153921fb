"""The host-side rules that choose kernels and launch shapes (no GPU needed)."""

import itertools

from llm_runtime_study_b200.ops import attention_bf16, gemm_bf16


def test_projection_kernel_choice_is_always_something_the_library_builds():
    for m, n, k in itertools.product((1, 17, 128, 129, 255, 256, 300, 512, 1000, 2048, 8192),
                                     (8, 264, 4096, 6144, 24576, 151936), (8, 72, 4096, 12288)):
        kernel, width = gemm_bf16.pick_kernel(m, n, k)
        assert kernel in gemm_bf16.KERNELS and width in (0, 128, 256)
        assert width == 256 or kernel == ("splitk" if width == 0 else "persistent")   # split-K chooses its own width
        if kernel == "pair":
            assert m >= gemm_bf16.PAIR_MIN_ROWS
        if kernel == "streamk":
            assert k >= 3072                                   # a K range long enough to share


def test_projection_kernel_choice_at_the_benchmark_shapes():
    layer = ((6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288))
    assert all(gemm_bf16.pick_kernel(2048, n, k) == ("pair", 256) for n, k in layer)
    assert gemm_bf16.pick_kernel(512, 4096, 4096) == ("persistent", 128)
    assert gemm_bf16.pick_kernel(256, 4096, 12288) == ("splitk", 0)
    assert gemm_bf16.pick_kernel(384, 4096, 12288) == ("streamk", 256)


def test_widths_of_the_pairs_tiles():
    """Rounds of tiles that are full or nearly so; 256 columns unless a narrower width is clearly ahead (host arithmetic)."""

    from llm_runtime_study_b200.ops import native

    width = lambda m, n, k=4096: native.query("b200_gemm_tcgen05_pair_width", m, n, k, 148)
    assert all(width(2048, n) == 256 for n in (4096, 6144, 24576)) and width(8192, 12288) == 256
    assert width(405, 24576) == 224 and width(405, 6144) == 192 and width(405, 4096) == 128 and width(1024, 6144) == 192
    for m in (256, 300, 700, 1500):
        for n in (16, 264, 5000, 151936):
            assert width(m, n) in (128, 192, 224, 256) and width(m, n, 1016) == 256
    assert gemm_bf16.pick_kernel(405, 6144, 4096) == gemm_bf16.pick_kernel(405, 4096, 12288) == ("pair", 256)
    assert gemm_bf16.pick_kernel(405, 6144, 1016) == ("persistent", 256)


def test_projections_to_few_columns():
    for k in (2048, 3072, 4096):
        assert gemm_bf16.pick_kernel(257, 1024, k) == gemm_bf16.pick_kernel(512, 1024, k) == ("splitk", 0)
        assert gemm_bf16.pick_kernel(513, 1024, k) == gemm_bf16.pick_kernel(2048, 264, k) == ("persistent", 128)


def test_projections_to_very_few_columns_share_only_long_k_ranges():
    for m in (257, 512):
        assert gemm_bf16.pick_kernel(m, 64, 2304) == gemm_bf16.pick_kernel(m, 96, 2048) == ("persistent", 128)
        assert gemm_bf16.pick_kernel(m, 64, 2560) == gemm_bf16.pick_kernel(m, 104, 2048) == ("splitk", 0)


def test_tiles_of_the_projections_by_features():
    """Whatever is chosen, the kernel takes it: widths in steps of 32 up to 256 each, shared K ranges only where they hold as many blocks."""

    for m, n, k in itertools.product((1, 32, 33, 129, 256, 257, 405, 512, 513, 1024, 1025, 2048, 16384), (8, 264, 1024, 4096, 6144, 12288), (8, 72, 200, 1024, 4096, 12288)):
        first, second, splits = gemm_bf16.features_shape(m, n, k, 148)
        assert first % 32 == 0 and 32 <= first <= 256 and second % 32 == 0 and 0 <= second <= first and splits in (1, 2, 4)
        assert splits <= -(-k // 64) and (splits == 1 or second == 0)
    assert gemm_bf16.features_shape(405, 4096, 4096, 148) == (224, 0, 2) and gemm_bf16.features_shape(1024, 4096, 4096, 148) == (256, 0, 1)
    assert gemm_bf16.features_shape(160, 1024, 2048, 148)[2] == 4


def test_accumulators_of_pairs_are_announced_only_to_a_wait():
    """Every arrival on a pair's accumulator barrier belongs to a later item that waits for it: the first use of a buffer waits for none."""

    from llm_runtime_study_b200.ops import native

    for items, stride, buffers in itertools.product((1, 2, 3, 4, 5, 73, 74, 75, 148, 149, 400), (1, 2, 18, 37, 74), (1, 2)):
        for cluster in range(min(items, stride)):
            mine = range(cluster, items, stride)
            arrivals, waits = [0] * buffers, [0] * buffers
            for local, item in enumerate(mine):
                waits[local % buffers] += local >= buffers
                arrivals[local % buffers] += native.query("b200_gemm_tcgen05_accumulator_reused", item, stride, buffers, items)
            assert arrivals == waits


def test_only_weights_at_rest_are_read_ahead(monkeypatch):
    """The operations wait for the kernel before; a model's projections, whose weights no kernel writes, need not."""

    import torch

    from llm_runtime_study_b200.ops import native
    from llm_runtime_study_b200.parts import Runtime
    from llm_runtime_study_b200.parts.linear import Projection

    asked = []
    monkeypatch.setattr(native, "require", lambda *a, **k: None)
    monkeypatch.setattr(native, "sm_count", lambda: 148)
    monkeypatch.setattr(native, "stream_ptr", lambda: None)
    monkeypatch.setattr(native, "call", lambda name, *args, **k: asked.append((name, args[-2])))
    w, b, rows = torch.zeros(4096, 2048).bfloat16(), torch.zeros(4096), lambda m: torch.zeros(m, 2048).bfloat16()
    gemm_bf16.linear(rows(405), w, None, torch.float32)
    gemm_bf16.linear_features(rows(64), w)
    gemm_bf16.linear_with_bias(rows(64), w, b)
    gemm_bf16.linear(rows(64), w, kernel="splitk")
    at_rest = len(asked)
    plain, biased = (Projection([w], biases, Runtime(torch.device("cpu"), torch.bfloat16)) for biases in (None, [b]))
    plain(rows(405), torch.float32), biased(rows(64)), plain(rows(200)), plain(rows(405), torch.float32, add_to=torch.zeros(405, 4096))
    assert [flag for _, flag in asked] == [0] * at_rest + [1] * (len(asked) - at_rest) and len(asked) == at_rest + 4
    assert {name for name, _ in asked} == {"b200_gemm_features", "b200_gemm_tcgen05"}


def test_which_projections_go_by_features():
    takes = gemm_bf16.by_features
    assert takes(405, 4096, 12288, True) and takes(129, 1024, 1024, True) and takes(1024, 4096, 4096, True) and takes(405, 4096, 4096, False)
    assert not takes(128, 4096, 4096, True) and not takes(2049, 4096, 4096, True) and not takes(256, 2048, 8192, True)
    assert not takes(405, 6144, 4096, False) and takes(640, 6144, 4096, False) and not takes(1024, 6144, 4096, False)


def test_a_wait_that_ran_out_is_reported_whichever_kernel_it_was_in(monkeypatch):
    import pytest

    from llm_runtime_study_b200.errors import KernelError
    from llm_runtime_study_b200.ops import native

    codes = {"b200_gemm_tcgen05_error": 0, "b200_gemm_features_error": 0}
    monkeypatch.setattr(native, "query", lambda name: codes[name])
    gemm_bf16.check_error()
    codes["b200_gemm_features_error"] = 5
    with pytest.raises(KernelError, match="by features.*shared tile"):
        gemm_bf16.check_error()
    codes.update(b200_gemm_tcgen05_error=2, b200_gemm_features_error=0)
    with pytest.raises(KernelError, match="projection: .*issue"):
        gemm_bf16.check_error()


def test_which_larger_projections_go_by_features():
    """Output heads and long K ranges: where the other kernels are ahead (timed both ways) they keep the product."""

    takes = gemm_bf16.by_features
    assert takes(512, 151936, 4096, True) and not takes(1024, 151936, 4096, True) and takes(1024, 151936, 1024, True)
    assert takes(640, 8192, 28672, True) and not takes(960, 8192, 28672, True) and takes(1024, 5120, 25600, True)
    assert not takes(256, 24576, 4096, True) and not takes(230, 12288, 16384, True) and takes(224, 24576, 4096, True) and takes(256, 32000, 4096, True)
    assert takes(200, 4096, 14336, False) and not takes(200, 4096, 20480, False) and takes(200, 5120, 25600, False)
    assert takes(640, 16384, 4096, False) and not takes(768, 16384, 4096, False) and takes(832, 16384, 4096, False) and not takes(896, 20480, 5120, False)
    assert takes(640, 5120, 25600, False) and not takes(704, 5120, 25600, False) and takes(832, 5120, 25600, False) and takes(704, 5120, 4096, False)


def test_gated_projections_of_some_rows_in_one_launch_where_the_weights_are_large():
    assert gemm_bf16.gated_in_one(24576, 4096) and gemm_bf16.gated_in_one(34816, 5120) and not gemm_bf16.gated_in_one(16384, 2048)


def test_gated_projections_of_few_or_short_rows_stay_with_the_library():
    """Products of as many weights that the split-K kernel takes longer for."""

    assert gemm_bf16.gated_in_one(51200, 5120) and gemm_bf16.gated_in_one(57344, 8192)
    for n, k in ((8192, 8192), (8192, 12288), (2048, 32768), (14336, 5120), (16384, 4096), (98304, 640), (65536, 1024), (49152, 2048)):
        assert not gemm_bf16.gated_in_one(n, k)


def test_decode_parts_are_bounded_and_use_the_gpu():
    for requests, kv_heads, longest, slots in itertools.product((1, 3, 8, 64, 500), (1, 8), (1, 100, 2048, 32768, 1 << 20), (296, 592)):
        parts = attention_bf16.decode_splits(requests, kv_heads, 1, longest, slots)
        assert 1 <= parts <= 64
        assert parts == 1 or longest // parts >= 64            # a part is never shorter than a few key blocks
    # parts that do not fit a cluster have to gain more than their meeting in memory costs
    assert attention_bf16.decode_splits(1, 8, 1, 2001, 296, together=8) == 8 and attention_bf16.decode_splits(1, 8, 1, 32768, 296, together=8) >= 16
    # one long sequence is cut into many parts, a full batch into none
    assert attention_bf16.decode_splits(1, 8, 1, 32768, 296) >= 16
    assert attention_bf16.decode_splits(64, 8, 1, 2048, 592) == 1
    assert attention_bf16.decode_splits(8, 8, 1, 2048, 296) == 4


def test_tile_map_orders_tiles_longest_first():
    table, count = attention_bf16.tile_map([5, 70, 1], 32, "cpu", kv_lens=[300, 70, 900])
    rows = table.t().tolist()                                    # [entry, first token, count]
    assert count == 5 and sorted(r[0] for r in rows) == [0, 1, 1, 1, 2]
    assert rows[0] == [2, 75, 1] and rows[1] == [0, 0, 5]        # 900 keys, then 300, then the 70-token prompt's tiles
    assert [r[2] for r in rows if r[0] == 1] == [6, 32, 32]      # its last tile (6 tokens, 70 keys) before the earlier ones


def test_few_rows_go_to_the_streaming_kernel_unless_the_weights_are_large():
    assert all(gemm_bf16.few_rows_kernel(m, 24576, 4096) == "skinny" for m in (1, 8))
    assert gemm_bf16.few_rows_kernel(1, 5120, 25600) == "splitk" and gemm_bf16.few_rows_kernel(8, 4096, 12288) == "skinny"
    assert gemm_bf16.few_rows_kernel(16, 24576, 4096) == "splitk" and gemm_bf16.few_rows_kernel(9, 51200, 5120) == "splitk"
    assert gemm_bf16.few_rows_kernel(16, 4096, 12288) == "skinny" and gemm_bf16.few_rows_kernel(16, 4096, 4096) == "skinny"


def test_split_k_shape_fills_the_sms_and_keeps_tiles_wide():
    """The width and cluster size the split-K kernel picks by itself (host arithmetic in the library)."""

    shape = gemm_bf16.splitk_shape
    assert shape(64, 4096, 4096) == (128, 4)           # 32 tiles x 4 = 128 CTAs on 148 SMs
    assert shape(16, 24576, 4096) == (192, 1)          # 128 tiles, nothing to share
    assert shape(16, 151936, 4096) == (224, 1)         # 679 tiles: 4.6 rounds of wide tiles, not 10.7 of narrow ones
    assert shape(200, 4096, 12288) == (256, 4)         # two row tiles: 32 wide tiles x 4 rather than 64 narrow ones x 2
    assert shape(8, 24, 64) == (256, 1)                # one K block cannot be shared
    for n, k in ((5120, 25600), (10240, 5120), (1000, 520), (7168, 5120)):
        width, splits = shape(16, n, k)
        assert width % 32 == 0 and 96 <= width <= 256 and splits in (1, 2, 4)
        assert -(-n // width) * splits <= 148 or splits == 1
        assert shape(128, n, k) == (width, splits)     # the choice does not depend on the rows that came along


def test_float32_tiles_go_by_the_gpus_own_number_of_multiprocessors():
    """1: few rows, 2 and 3: tiles of 64 and 128 rows, 4: short rows; by a B200's 148 and by fewer."""

    from llm_runtime_study_b200.ops import native

    choice = lambda m, n, k, sms=148, gated=0: native.query("b200_gemm_f32_choice", m, n, k, gated, sms)
    assert choice(8, 1024, 3072) == choice(24, 64, 64) == choice(1, 16, 4, gated=1) == 1 and choice(100, 16, 32) == 4
    assert choice(509, 6144, 1024) == 3 and choice(700, 4096, 1024) == choice(130, 6144, 1024) == choice(509, 1024, 3072) == 2
    assert choice(700, 4096, 1024, 100) == choice(509, 1024, 3072, 60) == 3 and choice(509, 6144, 1024, 60) == choice(9, 6400, 1024, 60) == 2 != choice(9, 6400, 1024)
    assert all(choice(m, 4096, 9000, sms) in (2, 3) for m in (33, 200, 3000) for sms in (1, 8, 30, 57, 148, 160))


def test_which_scans_go_in_chunks():
    from llm_runtime_study_b200.ops import sequence_state as S

    assert S.scans_in_chunks(2048, 1, 32, 128, False) and S.scans_in_chunks(405, 25, 32, 128, False)
    assert not S.scans_in_chunks(2048, 1, 32, 128, True)          # float32: sums that no cut changes
    assert not S.scans_in_chunks(2048, 1, 32, 136, False) and not S.scans_in_chunks(40, 1, 32, 128, False)
    assert not S.scans_in_chunks(1 << 20, 1, 32, 128, False)      # records of 57 GB
    assert S.scans_single(8, 8, 128, 64, False) and not S.scans_single(9, 8, 128, 64, False)
    assert S.scans_single(3, 3, 128, 64, False, [1, 1, 1]) and not S.scans_single(3, 3, 128, 64, False, [0, 2, 1])   # as many rows, another cut
    assert not S.scans_single(8, 8, 128, 33, False) and not S.scans_single(8, 8, 129, 64, False) and not S.scans_single(8, 8, 128, 64, True)


def test_records_of_long_portions_come_in_slices():
    from llm_runtime_study_b200.ops import sequence_state as S

    chunk = 32 * 27_136                      # 32 heads of 128, the delta rule
    fit = S.CHUNK_SLICE_BYTES // chunk
    assert S.chunk_slices([2048], 2048, 1, 128, chunk) == [(0, 2048, 128)]
    for lens in ([16_000], [5_000, 300, 9_001], [17_000, 1]):
        whole = sum(-(-m // 16) for m in lens)
        for known in (lens, None):
            slices = S.chunk_slices(known, sum(lens), len(lens), whole if known else sum(lens) // 16 + len(lens), chunk)
            assert max(held for _, _, held in slices) <= fit
            assert all(skip % 16 == most % 16 == 0 for skip, most, _ in slices)
            assert slices[-1][0] + slices[-1][1] >= max(lens) and [s[0] for s in slices[1:]] == [s[0] + s[1] for s in slices[:-1]]
            if known:
                assert sum(held for _, _, held in slices) == whole


def test_records_of_one_prompt_are_there_at_once():
    """With the size that the records have: prompts and batches up to some 2,400 tokens of 32 heads of 128 are one launch."""

    from llm_runtime_study_b200.ops import native
    from llm_runtime_study_b200.ops import sequence_state as S

    size = lambda dim, delta: native.query("b200_scan_chunks_record_floats", dim, delta) * 4
    assert size(128, 1) == 44_288 and size(128, 0) == 28_928
    for heads, dim, delta, lens in ((32, 128, 1, [2048]), (32, 128, 1, [800, 800, 800]), (32, 128, 0, [3700]), (64, 128, 0, [34] * 32), (64, 64, 1, [2300]), (64, 32, 0, [6300])):
        chunks = sum(-(-m // 16) for m in lens)
        assert len(S.chunk_slices(lens, sum(lens), len(lens), chunks, heads * size(dim, delta))) == 1
    assert len(S.chunk_slices([9000], 9000, 1, 563, 32 * size(128, 1))) > 1


def test_which_portions_go_in_chunks(monkeypatch):
    """By a portion's own length: many short ones beside each other, or single tokens beside a long one, are no reason."""

    from llm_runtime_study_b200.ops import sequence_state as S

    monkeypatch.setattr(S.native, "sm_count", lambda: 148)
    least = lambda lens, heads=32, dim=128, columns=128, delta=False: S.portion_in_chunks(lens, heads, dim, columns, delta)
    assert least([2] * 64) == least([7] * 8) == least([23] * 100) == least([47] * 100, delta=True) == 0
    assert least([30] * 8) == 24 and least([30] * 2) == least([30] * 8, heads=4) == 0
    assert least([1] * 24 + [381]) == least([2048], delta=True) == least([1, 300], delta=True) == 48
    assert least([300], heads=16) == least([1] * 24 + [300], heads=16) == 64 and least([300], heads=16, delta=True) == 96
    assert least([300], heads=4) == 64 and least([300, 1], heads=4) == 96 and least([300, 1], heads=4, delta=True) == 128
    assert least([100] * 64, heads=8, dim=64, columns=64) == 0 and least([100], heads=8, dim=64, columns=64) == 64
    assert S.scan_runs([1] * 24 + [381], 48) == [("single", 0, 24), ("chunks", 24, 25)]
    assert S.scan_runs([1, 2, 1, 0], 0) == [("chain", 0, 4)] and S.scan_runs([1, 1], 0) == [("single", 0, 2)]
    assert S.scan_runs([1, 900, 5, 1, 130, 128], 48) == [("single", 0, 1), ("chunks", 1, 2), ("chain", 2, 4), ("chunks", 4, 6)]
    assert S.scan_runs([1, 60, 3, 60], 48) == [("chain", 0, 4)] and S.scan_runs([1, 1, 60, 60], 48)[1] == ("chunks", 2, 4)
    assert S.scan_runs([900, 1] * 3, 48) == [("chain", 0, 6)]              # more launches than it is worth
    plan = lambda lens, n, entries, fixed=False: S._scan_plan(lens, n, entries, 32, 128, 128, 128, False, fixed)
    assert plan([1] * 24 + [381], 405, 25) == [("single", 0, 24), ("chunks", 24, 25)]
    assert plan([1] * 24 + [381], 405, 25, fixed=True) == [("chain", 0, 25)]
    assert plan(None, 405, 25) == [("chain", 0, 25)] and plan(None, 1200, 25) == [("chunks", 0, 25)] and plan(None, 8, 8) == [("chain", 0, 8)]


def test_short_portions_with_row_gates_go_in_chunks_where_they_fill_them(monkeypatch):
    """The normaliser is a 129th column, a block of its own: nearly two full chunks a portion, and no second round of CTAs that is nearly empty."""

    from llm_runtime_study_b200.ops import sequence_state as S

    monkeypatch.setattr(S.native, "sm_count", lambda: 148)
    least = lambda lens, heads, dim=128, columns=129: S.portion_in_chunks(lens, heads, dim, columns, False, True)
    assert least([24] * 8, 16) == least([27] * 32, 64) == 0 and least([28] * 8, 16) == least([34] * 6, 16) == 28
    assert least([32] * 4, 16) == least([32] * 16, 4) == least([32] * 8, 8) == 0 and least([48] * 4, 16) == 48      # 320 CTAs, two an SM
    assert least([40] * 32, 16, 96) == 0 and least([48] * 32, 16, 96) == 48
    assert S.portion_in_chunks([24] * 8, 16, 128, 128, False) == 24
    assert S._scan_plan([24] * 8, 192, 8, 16, 128, 128, 129, False, False) == [("chain", 0, 8)]
    assert S._scan_plan([24] * 8, 192, 8, 16, 128, 128, 128, False, False) == [("chunks", 0, 8)]


def test_parts_of_a_single_tokens_keys_over_shared_rows(monkeypatch):
    """Rows too wide for two CTAs a multiprocessor are cut into at most one round of CTAs, narrow ones into two."""

    from llm_runtime_study_b200.ops import attention_latent

    monkeypatch.setattr(attention_latent.native, "sm_count", lambda: 148)
    for requests in (1, 2, 7, 8, 74, 75, 148, 149, 300):
        for heads in (1, 32, 64, 65):
            ctas = requests * -(-heads // 64)
            wide = attention_latent.decode_splits(requests, heads, 1 << 20, 576)
            narrow = attention_latent.decode_splits(requests, heads, 1 << 20, 80)
            assert wide == 1 or wide == 32 or ctas * wide <= 148 < ctas * (wide + 1)
            assert narrow == 32 or ctas * narrow >= 296 > ctas * (narrow - 1)
            assert wide <= narrow
    # the exchange of scores counts (rows of 416 columns do not fit twice because of it), and so do the registers of many value columns
    assert attention_latent.two_fit(400, 128) and not attention_latent.two_fit(416, 128) and attention_latent.two_fit(80, 64)
    assert attention_latent.two_fit(208, 144) and not attention_latent.two_fit(208, 160)
    assert attention_latent.decode_splits(32, 16, 777, 320, 256) == 4 and attention_latent.decode_splits(32, 16, 777, 192, 128) == 6
    assert attention_latent.decode_splits(8, 32, 2049, 576) == 16
    assert attention_latent.decode_splits(1, 32, 511, 576) == 3 and attention_latent.decode_splits(1, 32, 100, 576) == 1
