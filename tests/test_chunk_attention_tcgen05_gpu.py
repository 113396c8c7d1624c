"""Attention with 32-bit weights in items of 128 rows (``csrc/attention_chunk_tcgen05.cu``): tiles of 64
keys, rows around 128, pages of every size that the kernel takes and one that it leaves to mma.sync,
the forms of the scores, infinities and NaN, missing pages."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

import test_kernels_gpu as kernels
import test_non_finite_gpu as non_finite
from gpu_helpers import PagedFixture

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("form", ["window", "slopes", "chunk"])
def test_forms(dim, form):
    kernels.test_chunk_attention_on_tensor_cores(dim, 128, form)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 3)])
def test_values_that_are_not_finite(dim, window, keep):
    non_finite.test_values_that_are_not_finite(dim, window, keep, 128, 1)


def _run(fx, qlen, heads, kv_heads, q, out, scale, status=0, **sight):
    from distengine_b200.kernels import recurrent as rk
    from distengine_b200.kernels.attention_plan import build_plan
    qlen = np.array(qlen, dtype=np.int32)
    pos0 = np.array(fx.kv_lens, dtype=np.int32) - qlen
    dim = fx.k_pages.shape[3]
    k_pages, v_pages, table = fx.to_device()
    ctx = SimpleNamespace(seq_slot=_t(np.array(fx.slots)), seq_qstart=_t(np.cumsum(qlen) - qlen),
                          seq_qlen=_t(qlen), seq_pos0=_t(pos0),
                          status=torch.zeros(1, dtype=torch.int32, device=DEV))
    items = _t(build_plan(qlen, pos0, heads // kv_heads, kv_heads, 128, 0, chunk=0).items)
    rk.chunk_attention(q, out, k_pages, v_pages, table, items, None, None, heads, kv_heads, dim, dim,
                       scale, 0, ctx, tile_rows=128, **sight)
    assert int(ctx.status.item()) == status
    return pos0


@pytest.mark.parametrize("dim,heads,kv_heads,page,window,keep,cap,odd", [
    (64, 4, 4, 8, None, 0, None, False), (128, 8, 2, 16, 200, 70, 3.0, False),
    (128, 5, 1, 64, None, 0, None, True), (64, 6, 2, 24, 130, 5, None, True),
    (128, 2, 2, 128, 64, 0, 50.0, False), (64, 16, 1, 4, 300, 1, None, False),
    (128, 3, 3, 32, 129, 64, None, False),
])
@pytest.mark.parametrize("gate", [None, "feature", "head"])
def test_pages_tiles_and_results(dim, heads, kv_heads, page, window, keep, cap, odd, gate):
    """Portions of up to 300 tokens behind up to 700 keys.  ``odd``: rows of q, the gate and the results
    at addresses and strides that no 16-byte access takes.  float32 results within the bound of float32
    sums of 700 terms; bfloat16 results are these rounded once."""
    lens, qlen = [700, 65, 129, 64, 1], [300, 65, 127, 1, 1]
    fx = PagedFixture(lens, kv_heads, dim, page, torch.bfloat16, DEV, seed=dim + page)
    if window:                              # pages that the first sequence's window has passed
        for p in range((keep + page - 1) // page, (400 - window + 1) // page):
            fx.block_table[fx.slots[0], p] = -1
    g = torch.Generator().manual_seed(page)
    n, pad = sum(qlen), 1 if odd else 0
    rows = torch.randn(n, heads * dim + 8 + pad, generator=g).to(torch.bfloat16).to(DEV)
    q = rows[:, pad: pad + heads * dim]
    gates = (torch.randn(n, heads * dim + 8 + pad, generator=g) * 2).to(torch.bfloat16).to(DEV)
    gates = gates[:, pad: pad + (heads if gate == "head" else heads * dim)]
    sink = torch.randn(heads, generator=g).to(DEV)
    got = {}
    for dtype in (torch.float32, torch.bfloat16):
        whole = torch.full((n, heads * dim + 8 + pad), 55.0, dtype=dtype, device=DEV)
        out = whole[:, pad: pad + heads * dim]
        pos0 = _run(fx, qlen, heads, kv_heads, q, out, dim ** -0.5, window=window or 0,
                    keep_first=keep, softcap=cap or 0.0, sink=sink, out_scale=0.75,
                    gate=gates if gate else None, gate_per_head=gate == "head")
        assert bool((whole[:, :pad] == 55.0).all()) and bool((whole[:, pad + heads * dim:] == 55.0).all())
        got[dtype] = out.double().cpu().view(n, heads, dim)
    assert torch.equal(got[torch.bfloat16], got[torch.float32].to(torch.bfloat16).double())
    at, q, gates, sink = 0, q.double().cpu().view(n, heads, dim), gates.double().cpu(), sink.double().cpu()
    for i, keys in enumerate(lens):
        pos, j = torch.arange(int(pos0[i]), keys), torch.arange(keys)
        seen = pos[:, None] >= j[None, :]
        if window:
            seen &= (pos[:, None] - j[None, :] < window) | (j < keep)[None, :]
        part = slice(at, at + qlen[i])
        at += qlen[i]
        for h in range(heads):
            kv = h * kv_heads // heads
            s = q[part, h] @ fx.k[i][:, kv].double().t() * dim ** -0.5
            s = cap * torch.tanh(s / cap) if cap else s
            e = torch.exp(s.masked_fill(~seen, float("-inf")))
            want = 0.75 * (e @ fx.v[i][:, kv].double()) / (e.sum(1, keepdim=True) + sink[h].exp())
            if gate == "head":
                want = want * torch.sigmoid(gates[part, h])[:, None]
            elif gate:
                want = want * torch.sigmoid(gates[part, h * dim: (h + 1) * dim])
            err = (got[torch.float32][part, h] - want).abs().max().item()
            assert err <= 4e-6 * max(1.0, want.abs().max().item()), (i, h, err)


@pytest.mark.parametrize("dim", [64, 128])
def test_seen_key_without_a_page(dim):
    """Status 2, and the rest of the keys as if the page's keys were not there."""
    fx = PagedFixture([300], 1, dim, 16, torch.bfloat16, DEV, seed=3)
    fx.block_table[fx.slots[0], 5] = -1
    q = torch.randn(300, 2 * dim, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    out = torch.empty(300, 2 * dim, device=DEV)
    _run(fx, [300], 2, 1, q.to(DEV), out, dim ** -0.5, status=2)
    j = torch.arange(300)
    seen = (j[:, None] >= j[None, :]) & ((j < 80) | (j >= 96))[None, :]
    for h in range(2):
        s = q[:, h * dim: (h + 1) * dim].double() @ fx.k[0][:, 0].double().t() * dim ** -0.5
        want = torch.softmax(s.masked_fill(~seen, float("-inf")), 1) @ fx.v[0][:, 0].double()
        err = (out[:, h * dim: (h + 1) * dim].double().cpu() - want).abs().max().item()
        assert err <= 4e-6 * max(1.0, want.abs().max().item()), (h, err)


@pytest.mark.parametrize("cap,low,high", [(1000.0, 0.05, 0.59), (1000.0, 0.61, 1.2), (300.0, 1.2, 3.0)])
def test_soft_cap(cap, low, high):
    """Two keys a token whose values are 1 and 0: the weights' logarithms give the difference of the two
    capped scores, in units of cap 2^-24.  Bound: the quotient's rounding, tanh to two units of its last
    place, the exponent's rounding, each time two, and the weights' own roundings."""
    n, dim, page = 600, 64, 16
    g = torch.Generator().manual_seed(3)
    x = ((torch.rand(n, generator=g) * (high - low) + low) * cap).to(torch.bfloat16).float()
    y = (x * (1 + 1 / 128)).to(torch.bfloat16).float()
    fx = PagedFixture([2] * n, 1, dim, page, torch.bfloat16, DEV)
    for i in range(n):
        fx.k[i].zero_(), fx.v[i].zero_()
        fx.k[i][0, 0, 0] = fx.k[i][1, 0, 1] = 1.0
        fx.v[i][0] = 1.0
    fx.rewrite()
    q = torch.zeros(n, dim)
    q[:, 0], q[:, 1] = x, y
    out = torch.empty(n, dim, device=DEV)
    _run(fx, [1] * n, 1, 1, q.to(torch.bfloat16).to(DEV), out, 1.0, softcap=cap)
    p = out[:, 0].cpu().double()
    clear = (p > 0.02) & (p < 0.98)             # (where the weights tell the difference)
    assert int(clear.sum()) > 100
    want = cap * (torch.tanh(x.double() / cap) - torch.tanh(y.double() / cap))
    units = (torch.log(p) - torch.log1p(-p) - want).abs() / (cap * 2.0 ** -24)
    assert units[clear].max().item() <= 2 * (0.5 + 2 + 0.5) + 1


@pytest.mark.parametrize("dim,heads,kv_heads", [(64, 4, 4), (128, 8, 2), (128, 3, 3), (64, 16, 1), (128, 5, 1)])
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("spoilt", [False, True])
def test_results_turned_back(dim, heads, kv_heads, gated, spoilt):
    """In the attention's own epilogue: the bits of float32 results that attention_finish then turns and
    gates, for one to 128 tokens a block, and in rows that are formed again."""
    from distengine_b200.kernels import recurrent as rk
    lens, qlen = [500, 131, 70], [300, 131, 1]
    fx = PagedFixture(lens, kv_heads, dim, 16, torch.bfloat16, DEV, seed=dim + heads)
    if spoilt:
        fx.v[0][450, 0, 5] = float("inf")
        fx.v[1][100, kv_heads - 1, dim - 1] = float("nan")
        fx.rewrite()
    g = torch.Generator().manual_seed(heads)
    n = sum(qlen)
    q = torch.randn(n, heads * dim, generator=g).to(torch.bfloat16).to(DEV)
    gate = torch.randn(n, heads * dim, generator=g).to(torch.bfloat16).to(DEV) if gated else None
    fv = torch.rand(dim // 2, generator=g).to(DEV)
    raw, want = torch.empty(n, heads * dim, device=DEV), torch.empty_like(q)
    pos0 = _run(fx, qlen, heads, kv_heads, q, raw, dim ** -0.5, window=200, keep_first=3)
    positions = _t(np.concatenate([np.arange(p, p + l) for p, l in zip(pos0, qlen)]))
    rk.attention_finish(raw, fv, gate, want, heads, dim, SimpleNamespace(positions=positions))
    out = torch.full_like(q, 9.0)
    _run(fx, qlen, heads, kv_heads, q, out, dim ** -0.5, window=200, keep_first=3, turned_back=fv, gate=gate)
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out.nan_to_num(1.0), want.nan_to_num(1.0))
    assert bool(want.isnan().any()) == spoilt


@pytest.mark.parametrize("dim", [64, 128])
def test_waits_that_run_out(dim, monkeypatch):
    """Every wait of the tiles' loop gives up at once: status 3, no result is stored, the copies in flight
    are waited for, and the launches after it find the GPU as before.  One to nine tiles a block."""
    from distengine_b200.kernels import library
    lens, qlen = [1100, 64, 130], [300, 64, 1]
    fx = PagedFixture(lens, 2, dim, 16, torch.bfloat16, DEV, seed=dim)
    q = torch.randn(sum(qlen), 6 * dim, generator=torch.Generator().manual_seed(dim))
    q = q.to(torch.bfloat16).to(DEV)
    want = torch.empty(sum(qlen), 6 * dim, device=DEV)
    _run(fx, qlen, 6, 2, q, want, dim ** -0.5)
    load = library.load
    monkeypatch.setattr(library, "load", lambda module, defines=(): load(
        module, ("ROLE_SPINS=0",) if module == "attention_chunk_tcgen05" else defines))
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.full_like(want, 55.0, dtype=dtype)
        _run(fx, qlen, 6, 2, q, out, dim ** -0.5, status=3)
        assert bool((out == 55.0).all())
    monkeypatch.undo()
    out = torch.full_like(want, 55.0)
    _run(fx, qlen, 6, 2, q, out, dim ** -0.5)
    assert torch.equal(out, want)
