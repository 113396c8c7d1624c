"""Decode steps in float32: rotation, cache write, attention and merge in one kernel, against the kernels
that it stands for: the same bits."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from gpu_helpers import PagedFixture, run_decode_attention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _apart(fx, qkv, heads, kv_heads, d, scale, window, inv_freq, rot, writes):
    """rope_kv_write, then the attention over its tiles of 8 rows and the merge."""
    from distengine_b200.kernels import ops
    from distengine_b200.kernels.attention import AttentionLauncher
    from distengine_b200.parts.context import StepPrep, Workspace
    n = len(fx.kv_lens)
    pos0 = np.array(fx.kv_lens, dtype=np.int32) - 1
    launcher = AttentionLauncher(torch.float32, heads, kv_heads, d, scale, window)
    prep = StepPrep(SimpleNamespace(seq_qlen=np.ones(n, dtype=np.int32), seq_pos0=pos0,
                                    seq_slot=np.array(fx.slots, dtype=np.int32)))
    launcher.prepare(prep, allow_decode=False)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    workspace = Workspace(torch.device(DEV))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(seq_slot=t(np.array(fx.slots)), seq_qstart=t(np.arange(n)),
                          seq_qlen=t(np.ones(n)), seq_pos0=t(pos0), notes=prep.notes, status=status,
                          arrays={k: t(v) for k, v in prep.extra.items()},
                          buffer=lambda name, shape, dt=None: workspace.get(name, shape,
                                                                            dt or torch.float32))
    assert not launcher.decode_step(ctx)
    k_pages, v_pages, table = fx.to_device()
    qkv = qkv.to(DEV)
    ops.rope_kv_write(qkv, t(pos0), t(np.array(fx.slots)), None if inv_freq is None else inv_freq.to(DEV),
                      rot, heads, kv_heads, d, k_pages, v_pages, table, writes, status)
    out = torch.full((n, heads * d), float("nan"), device=DEV)
    launcher.run(qkv, out, k_pages, v_pages, table, ctx)
    assert int(status.item()) == 0
    return out.cpu(), k_pages.cpu(), v_pages.cpu()


@pytest.mark.parametrize("heads,kv_heads,d,rot,page,window", [
    (32, 4, 64, 64, 16, None), (6, 2, 64, 32, 8, 70), (8, 1, 128, 128, 16, None), (3, 3, 128, 64, 4, 200),
    (5, 1, 256, 256, 16, None), (4, 4, 20, 12, 16, 33), (2, 1, 36, 0, 8, None), (7, 1, 252, 4, 32, 129),
])
@pytest.mark.parametrize("writes", [True, False])
@pytest.mark.parametrize("lens", [(1, 520, 33, 128), (129, 2, 64, 256, 257, 900), (31,) * 40])
def test_decode_attention_in_one_kernel(heads, kv_heads, d, rot, page, window, writes, lens):
    """Lengths around a tile's 32 keys and a range's 128, twice on the same buffers."""
    fx = PagedFixture(list(lens), kv_heads, d, page, torch.float32, DEV, seed=d)
    g = torch.Generator().manual_seed(heads + len(lens))
    qkv = torch.randn(len(lens), (heads + 2 * kv_heads) * d, generator=g)
    inv_freq = torch.rand(rot // 2, generator=g) if rot else None
    args = (heads, kv_heads, d, d ** -0.5, window, inv_freq, rot, writes)
    want = _apart(fx, qkv, *args)
    got = run_decode_attention(fx, qkv, *args, repeats=2)
    for a, b, name in zip(got, want, ("out", "k", "v")):
        assert torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0)), name     # (free pages hold NaN)
    assert torch.isfinite(got[0]).all()


@pytest.mark.parametrize("heads,kv_heads,d,window", [(32, 4, 64, None), (6, 2, 20, 9), (8, 1, 128, None), (3, 3, 256, 40)])
@pytest.mark.parametrize("lens,qlen", [((10, 32, 33, 1), (10, 17, 2, 1)), ((43,) * 9, (3,) * 9), ((200, 96), (5, 33))])
def test_tiles_of_8_rows_through_tiles_of_keys(heads, kv_heads, d, window, lens, qlen, monkeypatch):
    """Small portions by either kernel: the same bits, also where a range is cut and merged."""
    from distengine_b200.kernels import library
    from gpu_helpers import run_paged_attention
    fx = PagedFixture(list(lens), kv_heads, d, 16, torch.float32, DEV, seed=d)
    g = torch.Generator().manual_seed(heads)
    q = [torch.randn(n, heads, d, generator=g) for n in qlen]
    out = []
    for by_tiles in (0, 1):
        monkeypatch.setattr(library.load("attention_simt"), "de_attn_simt_by_tiles", lambda *sizes: by_tiles)
        for chunk in (0, 32, None):
            out.append(run_paged_attention(fx, q, heads, kv_heads, d, d ** -0.5, window, shape="rows8",
                                           chunk=chunk)[0])
    assert torch.isfinite(out[0]).all()
    for i in range(3):
        assert torch.equal(out[i], out[i + 3]), i
