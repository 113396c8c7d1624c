"""Infinities and NaN among the values: they reach the tokens that see them and no others, and an
infinity stays one.  Attention with 32-bit weights on the tensor cores, whose products take a whole
tile's values for a whole tile's tokens, and the read-outs of the chunked recurrences."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from gpu_helpers import PagedFixture
from test_chunked_recurrences_gpu import _step
from test_vomotar_mechanisms_gpu import _gen, _scan_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF, NAN = float("inf"), float("nan")
# (sequence, key, kv head, feature, value): before all tokens of the portions, inside a window's
# reach of some of them only, among the portions' own
BAD = [(0, 20, 0, 7, INF), (0, 101, 1, 2, -INF), (0, 150, 0, 3, INF), (0, 151, 0, 60, NAN),
       (0, 180, 1, 5, -INF), (1, 0, 1, 33, INF), (1, 60, 0, 0, NAN), (2, 128, 0, 9, INF)]


def _attend(fx, qlen, heads, kv_heads, dim, rows, window, keep):
    """The last ``qlen`` tokens of each sequence: float32 results [N, heads, dim]."""
    from distengine_b200.kernels import recurrent as rk
    from distengine_b200.kernels.attention_plan import build_plan
    qlen = np.array(qlen, dtype=np.int32)
    pos0 = np.array(fx.kv_lens, dtype=np.int32) - qlen
    n = int(qlen.sum())
    q = torch.randn(n, heads, dim, generator=_gen(dim)).to(torch.bfloat16)
    k_pages, v_pages, table = fx.to_device()
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    ctx = SimpleNamespace(n_seqs=len(qlen), seq_slot=t(np.array(fx.slots)),
                          seq_qstart=t(np.cumsum(qlen) - qlen), seq_qlen=t(qlen), seq_pos0=t(pos0),
                          status=torch.zeros(1, dtype=torch.int32, device=DEV))
    out = torch.full((n, heads * dim), 77.0, device=DEV)
    if rows:
        items = t(build_plan(qlen, pos0, heads // kv_heads, kv_heads, rows, 0, chunk=0).items)
        rk.chunk_attention(q.view(n, -1).to(DEV), out, k_pages, v_pages, table, items, None, None,
                           heads, kv_heads, dim, dim, dim ** -0.5, 0, ctx, tile_rows=rows,
                           window=window, keep_first=keep)
    else:
        rk.chunk_attention_decode(q.view(n, -1).to(DEV), out, k_pages, v_pages, table, None, None,
                                  heads, kv_heads, dim, dim, dim ** -0.5, 0, ctx, window=window,
                                  keep_first=keep)
    assert int(ctx.status.item()) == 0
    return q, pos0, out.double().cpu().view(n, heads, dim)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 3)])
@pytest.mark.parametrize("rows,copies", [(32, 1), (64, 1), (0, 1), (0, 30)])
def test_values_that_are_not_finite(dim, window, keep, rows, copies):
    """rows 0: single tokens, eight and four warps a block.  Bound of the finite results: as float32
    sums of up to 200 terms."""
    heads, kv_heads = 6, 2
    fx = PagedFixture([200, 70, 129] * copies, kv_heads, dim, 16, torch.bfloat16, DEV, seed=dim)
    for c in range(copies):
        for seq, key, head, feature, value in BAD:
            fx.v[3 * c + seq][key, head, feature] = value
    fx.rewrite()
    qlen = ([65, 37, 1] if rows else [1, 1, 1]) * copies
    q, pos0, got = _attend(fx, qlen, heads, kv_heads, dim, rows, window, keep)
    at, met = 0, 0
    for i, keys in enumerate(fx.kv_lens):
        for t in range(qlen[i]):
            pos = int(pos0[i]) + t
            j = torch.arange(keys)
            seen = j <= pos
            if window:
                seen &= (pos - j < window) | (j < keep)
            k = fx.k[i][seen].double().repeat_interleave(heads // kv_heads, 1)
            v = fx.v[i][seen].double().repeat_interleave(heads // kv_heads, 1)
            p = torch.softmax(torch.einsum("hd,jhd->hj", q[at + t].double(), k) * dim ** -0.5, 1)
            want = torch.einsum("hj,jhd->hd", p, v)
            assert torch.equal(got[at + t].isnan(), want.isnan()), (i, pos)
            infinite = want.isinf()
            assert torch.equal(got[at + t][infinite], want[infinite]), (i, pos)
            met += int((~want.isfinite()).sum())
            fine = want.isfinite()
            assert ((got[at + t] - want)[fine].abs() <= 4e-6 * want[fine].abs().max()).all(), (i, pos)
        at += qlen[i]
    assert met


@pytest.mark.parametrize("rule", ["delta", "decay", "decay-bf16"])
@pytest.mark.parametrize("value", [INF, NAN])
def test_chunks_with_a_value_that_is_not_finite(rule, value):
    """One head's value at one token of a portion: the same bits as without it but for that head's
    column from that token on, and that column not finite there."""
    from distengine_b200.kernels import recurrent as rk
    H, dk, dv, lens, slots = 2, 64, 128, (200, 193), (1, 0)
    ctx, items, portions, _ = _step(lens, slots)
    n, bad, head, col = sum(lens), 100, 1, 37
    flat = lambda t: t.reshape(n, -1).to(DEV).contiguous()
    q, k, v, beta, dec = _scan_inputs(n, H, H, dk, dv, 3)
    results = []
    for dirty in (False, True):
        vv = v.clone()
        if dirty:
            vv[bad, head, col] = value
        if rule == "decay-bf16":
            vv = vv.to(torch.bfloat16)
        state = torch.randn(2, H * dk * dv, generator=_gen(1)).to(DEV)
        out = torch.full((n, H * dv), 77.0, device=DEV)
        if rule == "delta":
            rk.delta_chunks(flat(q), flat(k), flat(vv), state, out, H, H, dk, dv, flat(dec),
                            flat(beta), items, portions, ctx)
        else:
            rk.decay_chunks(flat(q), flat(k), flat(vv), state, out, H, dk, dv,
                            torch.tensor([0.99, 0.9]).to(DEV), items, portions, ctx)
        results.append((out.cpu().view(n, H, dv), state.cpu().view(2, H, dk, dv)))
    (clean, clean_state), (got, got_state) = results
    reached = torch.zeros_like(clean, dtype=torch.bool)
    reached[bad: lens[0], head, col] = True
    assert torch.equal(got[~reached], clean[~reached])
    assert not got[reached].isfinite().any()
    kept = torch.ones_like(clean_state, dtype=torch.bool)
    kept[slots[0], head, :, col] = False
    assert torch.equal(got_state[kept], clean_state[kept])
    assert not got_state[~kept].isfinite().any()
