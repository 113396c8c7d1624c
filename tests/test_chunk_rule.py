"""When a recurrent layer's longer portions go through its states by chunks: decided from sizes and
lengths alone, so it can be checked without a GPU."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from distengine_b200.kernels import recurrent as rk
from distengine_b200.parts.recurrent import ChunkedMixer


def _prepared(lens):
    lens = np.asarray(lens, dtype=np.int32)
    notes = {}
    prep = SimpleNamespace(notes=notes, add=lambda name, array: None, host=SimpleNamespace(
        seq_qlen=lens, seq_qstart=(np.cumsum(lens) - lens).astype(np.int32)))
    ChunkedMixer.prepare(SimpleNamespace(), prep)
    return SimpleNamespace(notes=notes)


def _chunked(lens, heads, dim, delta, dtype=torch.bfloat16, dv=None, offset=0):
    dv = dv or dim
    mixer = SimpleNamespace(dtype=dtype, heads=heads, dk=dim, dv=dv)
    v = torch.zeros(4 * heads * dv + 4, dtype=torch.float32)[offset: offset + 2 * heads * dv].view(2, -1)
    return ChunkedMixer.chunked(mixer, _prepared(lens), v, torch.zeros(2, heads * dim * dv), delta)


# (portions, heads, size, by chunks?), measured on B200 both ways
DELTA = [((2048,), 16, 128, True), ((512,), 16, 128, True), ((200,) * 10, 16, 128, True),
         ((200,) * 32, 16, 128, False), ((200,) * 10, 64, 128, False), ((256,) * 10, 64, 64, False),
         ((2048,), 64, 128, True), ((1000, 1000), 16, 64, True), ((500,) * 4, 64, 64, True),
         ((512,), 16, 64, True), ((192,), 16, 128, False), ((256,), 8, 64, False),
         ((200,) * 10, 16, 64, False), ((200,) * 32, 16, 64, False), ((200,) * 10, 64, 64, False),
         ((400,) * 10, 64, 64, False), ((200,) * 4, 16, 64, False)]
DECAY = [((2048,), 16, 128, True), ((256,), 16, 128, True), ((512,), 8, 64, True),
         ((200,) * 10, 64, 64, True), ((192,), 64, 64, True), ((200,), 8, 64, False),
         ((256,), 16, 64, False), ((200,) * 4, 8, 64, False), ((320,), 8, 64, False),
         ((192,), 8, 128, False), ((192,), 16, 128, True)]


@pytest.mark.parametrize("lens,heads,dim,chunks", DELTA)
def test_delta_rule(lens, heads, dim, chunks):
    assert _chunked(lens, heads, dim, True) == (1 if chunks else 0)


@pytest.mark.parametrize("lens,heads,dim,chunks", DECAY)
def test_decay_per_head(lens, heads, dim, chunks):
    assert _chunked(lens, heads, dim, False) == (1 if chunks else 0)


def test_the_kernels_sizes():
    """The plan's chunk and the sizes that go by chunks are those of the kernels."""
    from distengine_b200.kernels import library
    lib = library.load("recurrent_chunks")
    assert lib.de_chunk_tokens() == rk.CHUNK
    for dk in (32, 64, 96, 128, 256):
        for dv in (32, 64, 96, 128, 192):
            assert bool(lib.de_chunk_ok(dk, dv)) == rk.chunks_ok(dk, dv)


def test_what_stays_with_the_scan():
    long = (2048,)
    assert _chunked(long + (5,), 16, 128, True) == 2          # the short one beside it
    assert _chunked(long, 16, 128, True, dtype=torch.float32) == 0
    assert _chunked((191, 191), 16, 128, True) == 0
    assert _chunked(long, 16, 96, True) == 0                  # key sizes 64 and 128 only
    assert _chunked(long, 16, 128, True, dv=96) == 0          # values in whole 64s
    assert _chunked(long, 16, 128, True, offset=1) == 0       # not in whole 16-byte pieces
