"""The host-side planning of attention work: items, chunks, the decode kernel's split.  No GPU."""

import numpy as np
import pytest

from distengine_b200.kernels.attention_plan import build_plan, choose_chunk, choose_decode_split

SMS = 148          # the planners are told the device's number of SMs; the tests plan for this many


def _covered(items, group, rows_per_tile):
    """(seq, row) -> sorted list of key ranges, from the items of a plan."""
    out = {}
    for seq, row0, begin, end, *_ in items.tolist():
        if begin >= end:
            continue
        out.setdefault((seq, row0), []).append((begin, end))
    return {k: sorted(v) for k, v in out.items()}


@pytest.mark.parametrize("window", [0, 37])
@pytest.mark.parametrize("chunk,cap", [(0, None), (64, None), (128, 6), (None, None)])
def test_every_row_tile_gets_its_keys_exactly_once(window, chunk, cap):
    qlen = np.array([130, 1, 1, 21, 2], dtype=np.int32)
    pos0 = np.array([0, 0, 76, 279, 31], dtype=np.int32)
    group, kv_heads, rows = 3, 2, 16
    plan = build_plan(qlen, pos0, group, kv_heads, rows, window, chunk, cap, sm_count=SMS)
    ranges = _covered(plan.items, group, rows)
    for seq in range(len(qlen)):
        rows_total = int(qlen[seq]) * group
        for row0 in range(0, rows_total, rows):
            last_row = min(row0 + rows, rows_total) - 1
            hi = int(pos0[seq]) + last_row // group + 1
            lo = max(0, int(pos0[seq]) + row0 // group - window + 1) if window else 0
            got = ranges[(seq, row0)]
            # chunks are disjoint, in order, and reach from at most lo to exactly hi
            assert got[0][0] <= lo and got[-1][1] == hi
            for (b0, e0), (b1, e1) in zip(got, got[1:]):
                assert e0 == b1
    if cap is not None:
        tiles = sum(-(-int(q) * group // rows) for q in qlen)
        assert plan.items.shape[0] == tiles * cap           # a fixed number of items per tile


def test_items_carry_their_tile_and_start_longest_first():
    qlen = np.array([64, 8, 300], dtype=np.int32)
    pos0 = np.array([0, 500, 0], dtype=np.int32)
    plan = build_plan(qlen, pos0, 2, 1, 16, 0, chunk=0)
    keys = plan.items[:, 3] - plan.items[:, 2]
    assert (np.diff(keys) <= 0).all()                       # falling number of keys
    assert sorted(plan.items[:, 7].tolist()) == list(range(plan.items.shape[0]))
    split = build_plan(qlen, pos0, 2, 1, 16, 0, chunk=128, sort=False)
    for tile in np.unique(split.items[:, 7]):
        mine = split.items[split.items[:, 7] == tile]
        live = mine[mine[:, 3] > mine[:, 2]]
        assert (mine[:, 6] == len(live)).all()              # chunks that hold keys
        if len(live) > 1:
            assert (live[:, 4] == live[0, 5] + np.arange(len(live))).all()   # partial slots in a row


def test_capped_plan_refuses_a_range_that_needs_more_chunks():
    with pytest.raises(ValueError, match="capped"):
        build_plan(np.array([1], dtype=np.int32), np.array([999], dtype=np.int32), 1, 1, 16, 0,
                   chunk=64, chunks_cap=4)


@pytest.mark.parametrize("tiles,kv_heads,span", [(8, 4, 1024), (1, 4, 1024), (64, 4, 1024), (8, 4, 64),
                                                 (1, 4, 32768), (8, 4, 32768), (256, 8, 2048),
                                                 (1, 1, 1), (3, 5, 100000)])
@pytest.mark.parametrize("per_sm", [4, 3, 2])
def test_decode_split_covers_the_span_with_whole_tiles_of_keys(tiles, kv_heads, span, per_sm):
    cluster, clusters, chunk = choose_decode_split(tiles, kv_heads, span, per_sm=per_sm, sm_count=SMS)
    assert 1 <= cluster <= 8 and clusters >= 1
    # one round of blocks over the SMs, unless even single blocks do not fit in one
    assert cluster == 1 or tiles * kv_heads * cluster <= per_sm * SMS
    assert chunk % 64 == 0 and chunk >= 64
    assert cluster * clusters * chunk >= span                # every key has an item
    assert chunk <= 2048 + 63                                # no block walks more than that
    if cluster > 1:
        assert span >= 64 * cluster // 2                     # no cluster of blocks without keys


def test_decode_split_takes_sizes_between_the_powers_of_two():
    # 64 tiles of one kv head each... 8 kv heads, three blocks an SM: 6 blocks a cluster fit, 8 not
    assert choose_decode_split(8, 8, 4096, per_sm=3, sm_count=SMS)[0] == 6
    assert choose_decode_split(8, 8, 4096, per_sm=4, sm_count=SMS)[0] == 8
    assert choose_decode_split(8, 4, 520, per_sm=4, sm_count=SMS)[0] == 8
    assert choose_decode_split(64, 4, 520, per_sm=4, sm_count=SMS)[0] == 2
    assert choose_decode_split(20, 4, 520, per_sm=4, sm_count=SMS)[0] == 4       # short ranges: powers of two


def test_clusters_of_eight_only_while_a_fifth_of_the_places_stays_free():
    # 4 kv heads, 4 blocks an SM: 592 places; clusters of 8 up to 473 blocks (14 sequences: 448)
    for sequences, want in ((8, 8), (12, 8), (14, 8), (15, 4), (16, 4), (18, 4), (32, 4), (37, 4),
                            (38, 2), (64, 2)):
        assert choose_decode_split(sequences, 4, 640, per_sm=4, sm_count=SMS)[0] == want, sequences


def test_chunk_choice_fills_the_gpu_or_leaves_ranges_whole():
    assert choose_chunk(1000, 4, 4096, sm_count=SMS) == 0                  # enough tiles: no split
    c = choose_chunk(8, 4, 4096, sm_count=SMS)
    assert c in (2048, 1024, 512, 256, 128, 64) and 8 * 4 * -(-4096 // c) >= 2 * SMS


@pytest.mark.parametrize("qlen,pos0,heads,kv_heads,dim,shape", [
    ([5], [0], 32, 4, 64, "rows8"), ([17] * 4, [0] * 4, 32, 4, 60, "rows8"), ([100], [0], 32, 4, 64, "rows8"),
    ([200], [0], 32, 4, 64, "rows32"), ([400], [0], 8, 8, 64, "rows32"), ([100], [1000], 8, 8, 128, "rows32"),
    ([17] * 4, [0] * 4, 32, 4, 256, "rows32"), ([17], [0], 8, 8, 256, "rows8")])
def test_float32_tiles_by_the_blocks_of_a_step(qlen, pos0, heads, kv_heads, dim, shape):
    """Small float32 steps take tiles of 8 rows, larger ones tiles of 32; single tokens beside a portion
    tiles of 8 either way; a step shaped for replay decides by its shape alone."""
    from types import SimpleNamespace

    import torch

    from distengine_b200.kernels.attention import AttentionLauncher
    from distengine_b200.parts.context import StepPrep
    launcher = AttentionLauncher(torch.float32, heads, kv_heads, dim, 1.0, None)
    for more in ([], [1]):
        arrays = []
        for graph_shape, start in ((None, 0), ({"context_cap": 1536}, 0), ({"context_cap": 1536}, 100)):
            host = SimpleNamespace(seq_qlen=np.array(qlen + more, dtype=np.int32),
                                   seq_pos0=np.array(pos0 + more, dtype=np.int32) + start)
            prep = StepPrep(host, graph_shape)
            launcher.prepare(prep)
            count = {s.name: prep.extra[f"{launcher.key}/{s.name}/items"] for s in launcher.shapes}
            arrays.append({name: a.shape for name, a in count.items()})
            if graph_shape is None:
                assert len(count[shape]) and (shape == "rows8" or bool(len(count["rows8"])) == bool(more))
                assert shape == "rows32" or not len(count["rows32"])
        assert arrays[1] == arrays[2]



@pytest.mark.parametrize("graph_shape", [None, {"context_cap": 1536}])
def test_float32_decode_steps_bring_no_list_of_merges(graph_shape):
    """The one-launch kernel merges by its items; the kernels apart need the list."""
    from types import SimpleNamespace

    import torch

    from distengine_b200.kernels.attention import AttentionLauncher
    from distengine_b200.parts.context import StepPrep
    launcher = AttentionLauncher(torch.float32, 32, 4, 64, 1.0, None)
    host = SimpleNamespace(seq_qlen=np.ones(3, dtype=np.int32), seq_slot=np.arange(3, dtype=np.int32),
                           seq_pos0=np.array([5, 700, 1200], dtype=np.int32))
    for fused in (True, False):
        prep = StepPrep(host, graph_shape)
        launcher.prepare(prep, allow_decode=fused)
        assert (prep.notes[launcher.key + "/decode"] is not None) == fused
        assert (len(prep.extra[f"{launcher.key}/rows8/combine"]) == 0) == fused


@pytest.mark.parametrize("dim,blocks,keys,by_tiles", [
    (64, 4, 10, 1), (64, 480, 17, 1), (64, 2000, 32, 1), (64, 400, 33, 0), (64, 480, 43, 1), (64, 480, 96, 1),
    (64, 480, 97, 0), (64, 700, 64, 0), (64, 1000, 64, 1), (128, 100, 32, 1), (128, 300, 32, 0), (128, 500, 20, 1),
    (128, 500, 33, 0), (256, 100, 32, 1), (256, 149, 32, 0), (256, 10, 33, 0), (32, 460, 50, 1), (32, 400, 50, 0),
    (66, 4, 10, 0)])
def test_float32_tiles_of_8_rows_over_few_keys(dim, blocks, keys, by_tiles):
    """Up to 32 keys, and up to 96 where it saves a round of blocks, tiles of 8 rows go through tiles of keys."""
    from distengine_b200.kernels import library
    assert library.load("attention_simt").de_attn_simt_by_tiles(dim, blocks, keys) == by_tiles


def test_the_plan_says_how_tiles_of_8_rows_go():
    from types import SimpleNamespace

    import torch

    from distengine_b200.kernels.attention import AttentionLauncher
    from distengine_b200.parts.context import StepPrep
    for dim, qlen, pos0, note in ((64, [10], [0], True), (64, [10], [500], False), (64, [3] * 40, [40] * 40, True),
                                  (128, [3] * 40, [40] * 40, False), (64, [200], [0], None), (18, [10], [0], None)):
        launcher = AttentionLauncher(torch.float32, 32, 4, dim, 1.0, None)
        prep = StepPrep(SimpleNamespace(seq_qlen=np.array(qlen, dtype=np.int32),
                                        seq_pos0=np.array(pos0, dtype=np.int32)))
        launcher.prepare(prep)
        assert prep.notes.get(launcher.key + "/by_tiles") is note
