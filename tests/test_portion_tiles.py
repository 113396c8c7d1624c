"""Rows of a tile of the attention with 32-bit weights, chosen from a step's lengths and the cache's page
size alone, so it can be checked without a GPU (the kernel libraries are loaded, none of them runs)."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from distengine_b200.kernels import recurrent as rk
from distengine_b200.parts.context import StepPrep


def _prep(qlen, pos0, page, graph_shape=None):
    host = SimpleNamespace(seq_qlen=np.array(qlen, dtype=np.int32),
                           seq_pos0=np.array(pos0, dtype=np.int32))
    return StepPrep(host, graph_shape, page)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("qlen,pos0", [([9], [1900]), ([500], [0]), ([2048], [0]), ([30] * 4, [500] * 4),
                                       ([300] + [1] * 20, [0] + [600] * 20), ([100], [0])])
def test_pages_that_the_kernel_takes_and_others(dim, qlen, pos0, monkeypatch):
    monkeypatch.setattr(rk, "_sms", lambda: 148)
    host = _prep(qlen, pos0, None).host
    without = rk.chunk_rows_per_tile(torch.bfloat16, dim, dim, True,
                                     rk.long_portion_rows(host.seq_qlen, 16, 4))
    for shape in (None, {"context_cap": 2048}):
        for page in (1, 2, 4, 12, 20, 8, 16, 24, 64):
            rows = rk.portion_tile_rows(torch.bfloat16, dim, dim, _prep(qlen, pos0, page, shape), 16, 4)
            assert rows == (128 if page % 8 == 0 else without), page
        assert rk.portion_tile_rows(torch.bfloat16, dim, dim, _prep(qlen, pos0, None, shape), 16, 4) == 128
    assert without in (32, 64)
    for dtype, size in ((torch.float32, dim), (torch.bfloat16, 96)):
        rows = rk.portion_tile_rows(dtype, size, size, _prep(qlen, pos0, 16), 16, 4)
        assert rows == rk.chunk_rows_per_tile(dtype, size, size, True,
                                              rk.long_portion_rows(host.seq_qlen, 16, 4))


@pytest.mark.parametrize("page", [4, 16])
def test_a_steps_plan_knows_its_page_size(page, monkeypatch):
    """``StepRunner`` tells the parts what pages its cache has."""
    from distengine_b200.engine import step
    from distengine_b200.kernels import ops
    seen = []
    monkeypatch.setattr(ops, "require_device", lambda device: None)
    monkeypatch.setattr(torch.cuda, "Event", lambda: None)
    monkeypatch.setattr(step.StepRunner, "_stage", lambda self, host, prep: ({}, [], 0, []))
    model = SimpleNamespace(device=torch.device("cpu"), dtype=torch.float32,
                            config=SimpleNamespace(vocabulary=10),
                            prepare=lambda prep: seen.append(prep.page_size))
    cache = SimpleNamespace(page_size=page, bindings=lambda: [], has=lambda r: True, reserve=lambda r: None,
                            length=lambda r: 0, slot=lambda r: 0)
    step.StepRunner(model, cache).prepare([step.StepEntry("a", [1, 2])])
    assert seen == [page]


# (tokens, position of the first, plain scores?, heads, key/value heads, size, tiles of 128 rows?), measured on B200
MEASURED = [
    ([2], [0], True, 16, 4, 128, False), ([64], [0], True, 16, 4, 128, False), ([96], [0], True, 16, 4, 128, True),
    ([96], [0], False, 16, 4, 128, False), ([200], [0], False, 16, 4, 128, True), ([9], [1900], True, 16, 4, 128, True),
    ([64] * 16, [0] * 16, True, 16, 4, 128, True), ([160] * 8, [0] * 8, True, 16, 4, 128, False),
    ([512] * 4, [0] * 4, False, 16, 4, 128, True), ([2] + [1] * 60, [50] + [400] * 60, True, 16, 4, 128, False),
    ([2] * 4, [160] * 4, False, 16, 4, 128, False), ([2048], [0], False, 16, 4, 128, True),
    ([1201, 1172], [0, 0], True, 16, 4, 128, True), ([2] * 16, [0] * 16, True, 16, 4, 64, False),
    ([96], [0], True, 16, 4, 64, True), ([200], [0], False, 16, 4, 64, False), ([512], [0], False, 16, 4, 64, True),
    ([9], [500], False, 16, 4, 64, False), ([9], [500], True, 16, 4, 64, True),
    ([2] + [1] * 30, [50] + [400] * 30, False, 12, 4, 64, False), ([2] * 64, [300] * 64, True, 16, 2, 64, False),
]


@pytest.mark.parametrize("qlen,pos0,plain,heads,kv_heads,dim,wide", MEASURED)
def test_tiles_of_128_rows_where_they_are_sooner(qlen, pos0, plain, heads, kv_heads, dim, wide, monkeypatch):
    monkeypatch.setattr(rk, "_sms", lambda: 148)
    rows = rk.portion_tile_rows(torch.bfloat16, dim, dim, _prep(qlen, pos0, 16), heads, kv_heads, plain)
    assert (rows == 128) == wide


def test_keys_out_of_a_windows_reach_do_not_count(monkeypatch):
    monkeypatch.setattr(rk, "_sms", lambda: 148)
    for reach, wide in ((0, True), (1024, True), (100, True), (20, False)):
        rows = rk.portion_tile_rows(torch.bfloat16, 128, 128, _prep([40], [1900], 16), 16, 4, True, reach)
        assert (rows == 128) == wide, reach


def test_a_launch_that_is_saved_counts_where_steps_go_launch_by_launch(monkeypatch):
    monkeypatch.setattr(rk, "_sms", lambda: 148)
    for qlen, pos0, plain, eager, replayed in (([33], [0], True, True, False), ([2048], [0], True, True, True),
                                               ([2] + [1] * 60, [50] + [400] * 60, True, False, False),
                                               ([2] + [1] * 30, [50] + [100] * 30, False, False, False)):
        for shape, wide in ((None, eager), ({"context_cap": 2048}, replayed)):
            rows = rk.portion_tile_rows(torch.bfloat16, 128, 128, _prep(qlen, pos0, 16, shape), 16, 4, plain,
                                        finishes=True)
            assert (rows == 128) == wide, (qlen, shape)
