"""float32 attention with infinities and NaN among queries, keys and values: they reach the rows that see
them and no others, in tiles of either height, in ranges cut or whole and in the one-launch decode kernel."""

import pytest
import torch

from gpu_helpers import PagedFixture, run_decode_attention, run_paged_attention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF, NAN = float("inf"), float("nan")
LENS, QLEN = (300, 70, 33, 1), (40, 70, 1, 1)


def _spoil(fx, what):
    if what == "a tile of keys":
        fx.k[0][224:256] = NAN
    elif what == "one key":
        fx.k[0][270, 0, 1] = NAN
        fx.k[1][0] = NAN
    elif what == "infinite keys":
        fx.k[0][265, 0] = INF
        fx.k[1][3, 0, 0] = -INF
    elif what == "values":
        fx.v[0][40, 0, 2], fx.v[1][50, 0, 0], fx.v[3][0, 0, 1] = INF, NAN, -INF
    fx.rewrite()


def _want(fx, q, heads, kv_heads, window):
    out = []
    for i, n in enumerate(fx.kv_lens):
        for t in range(q[i].shape[0]):
            pos, j = n - q[i].shape[0] + t, torch.arange(n)
            seen = (j <= pos) & (j > pos - (window or n))
            k = fx.k[i][seen].double().repeat_interleave(heads // kv_heads, 1)
            v = fx.v[i][seen].double().repeat_interleave(heads // kv_heads, 1)
            s = torch.einsum("hd,jhd->hj", q[i][t].double(), k) * q[i].shape[2] ** -0.5
            e = torch.exp(s - s.max(1, keepdim=True)[0])
            out.append(torch.einsum("hj,jhd->hd", e, v) / e.sum(1)[:, None])
    return torch.stack(out)


def _close(got, want, what):
    # (where a row is not finite: NaN if the exact result is, an infinity of its sign otherwise)
    assert torch.equal(got.isnan(), want.isnan()), what
    assert torch.equal(got[want.isinf()], want[want.isinf()]), what
    fine = want.isfinite()
    assert ((got - want)[fine].abs() <= 4e-6 * want[fine].abs().max()).all(), what


@pytest.mark.parametrize("dim,window", [(64, None), (64, 50), (20, None), (128, 40), (256, None), (18, None)])
@pytest.mark.parametrize("what", ["a tile of keys", "one key", "infinite keys", "values", "a query"])
def test_what_is_not_finite_reaches_the_rows_that_see_it(dim, window, what):
    """Bound of the finite results: as float32 sums of up to 300 terms."""
    heads, kv_heads = 4, 1
    g = torch.Generator().manual_seed(dim)
    fx = PagedFixture(list(LENS), kv_heads, dim, 16, torch.float32, DEV, seed=dim)
    _spoil(fx, what)
    q = [torch.randn(n, heads, dim, generator=g) for n in QLEN]
    if what == "a query":
        q[0][7, 1, 3], q[1][0, 2] = NAN, NAN
        q[3][0] = NAN
    want = _want(fx, q, heads, kv_heads, window)
    assert bool((~want.isfinite()).any())
    for shape in ("rows8", "rows32") if dim % 4 == 0 else ("rows8",):
        for chunk in (0, 64, None):
            got, _ = run_paged_attention(fx, q, heads, kv_heads, dim, dim ** -0.5, window, chunk=chunk,
                                         shape=shape)
            _close(got.double().view(-1, heads, dim), want, (shape, chunk))
    if dim % 4 or what == "a query":         # (that helper compares the rows before and after)
        return
    # the last tokens as a decode step, the newest key and value the token's own
    last = torch.stack([t[-1] for t in q])
    own = [torch.stack([t[-1] for t in of]) for of in (fx.k, fx.v)]
    qkv = torch.cat([t.flatten(1) for t in (last, *own)], 1)
    got = run_decode_attention(fx, qkv, heads, kv_heads, dim, dim ** -0.5, window, None, 0, True)[0]
    ends = torch.tensor(QLEN).cumsum(0) - 1
    _close(got.double().view(-1, heads, dim), want[ends], "decode")
