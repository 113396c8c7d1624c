"""When a step's queries, keys and values are prepared in runs of tokens: decided from sizes alone, so it can
be checked without a GPU."""

import pytest
import torch

from distengine_b200.kernels import library
from distengine_b200.kernels.ops import _tag

# (heads of q, k and v, head size, taps, dtype, tokens that go a token a block, tokens that go in runs),
# measured on B200 both ways
MEASURED = [
    (24, 128, False, torch.bfloat16, (127, 128, 650, 700), (300, 400, 511, 512, 560, 592, 750, 800, 1000, 2048)),
    (20, 128, False, torch.bfloat16, (128, 200, 600, 650, 700), (300, 400, 512, 592, 750, 888, 1500)),
    (16, 128, False, torch.bfloat16, (128, 200), (300, 400, 512, 600, 700, 900, 2048)),
    (12, 128, False, torch.bfloat16, (128, 200, 300), (400, 500, 512, 600, 700, 888, 900)),
    (48, 128, False, torch.bfloat16, (127,), (128, 300, 512, 600, 650, 700, 1200)),
    (24, 64, False, torch.bfloat16, (127,), (128, 300, 512, 650, 700, 900)),
    (48, 64, False, torch.bfloat16, (127,), (128, 512, 600, 700)),
    (24, 128, False, torch.float32, (127,), (128, 512, 600, 700)),
    (24, 128, True, torch.bfloat16, (127,), (128, 512, 600, 700, 2048)),
    (12, 64, True, torch.bfloat16, (127,), (128, 600, 1200)),
]


@pytest.mark.parametrize("heads,dim,taps,dtype,single,runs", MEASURED)
def test_runs_where_they_are_sooner(heads, dim, taps, dtype, single, runs):
    in_runs = library.load("attention_chunk").de_qkv_prepare_in_runs
    for tokens, want in [(n, 0) for n in single] + [(n, 1) for n in runs]:
        assert in_runs(_tag(dtype), tokens, heads, dim, int(taps), 148) == want, tokens
