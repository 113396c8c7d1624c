"""The kernels before and after the window and sink attention that take four features at a time
against their general forms, which rows at other addresses reach: the same bits."""

import pytest
import torch

from test_vomotar_mechanisms_gpu import _ctx, _gen

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rows(t, pad):
    """The same rows, `pad` elements apart beyond their own."""
    wide = torch.zeros(t.shape[0], t.shape[1] + pad, dtype=t.dtype, device=DEV)
    wide[:, : t.shape[1]] = t.to(DEV)
    return wide[:, : t.shape[1]]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,rot,turned", [(3, 1, 64, 64, 64, True), (4, 2, 128, 40, 32, True),
                                                   (2, 2, 12, 4, 8, False), (8, 4, 256, 256, 256, True),
                                                   (1, 1, 20, 12, 0, False)])
@pytest.mark.parametrize("write", [True, False])
def test_rotation_and_cache_write(dtype, H, G, dk, dv, rot, turned, write):
    from distengine_b200.kernels import recurrent as rk
    lens, page, g = (5, 1, 9), 8, _gen(dk)
    ctx = _ctx(lens, (3, 900, 0), (1, 0, 2))
    n = sum(lens)
    proj = torch.randn(n, H * dk + G * (dk + dv), generator=g).to(dtype)
    fk, fv = torch.rand(rot // 2, generator=g), torch.rand(dv // 2, generator=g)
    table = torch.full((3, 120), -1, dtype=torch.int32)
    table[1, 0], table[0, 112], table[2, 0], table[2, 1] = 2, 0, 3, 1
    results = []
    for pad in (4 - proj.shape[1] % 4, 5 - proj.shape[1] % 4):      # whole groups of four, or not
        p = _rows(proj, pad)
        kp = torch.zeros(4, G, page, dk, dtype=dtype, device=DEV)
        vp = torch.zeros(4, G, page, dv, dtype=dtype, device=DEV)
        rk.kv_write_rotated(p, fk.to(DEV), rot, fv.to(DEV) if turned else None, H, G, dk, dv, kp, vp,
                            table.to(DEV), write, ctx)
        # (the second sequence's position 900 has its page; one of the first's does not matter)
        o = torch.randn(n, H * dv, generator=_gen(1)).to(DEV)
        gate = torch.randn(n, H * dv, generator=_gen(2)).to(dtype)
        out = torch.empty(n, H * dv, dtype=dtype, device=DEV)
        rk.attention_finish(o, fv.to(DEV) if turned else None, _rows(gate, 4 if pad % 2 == 0 else 5),
                            out, H, dv, ctx)
        results.append((p.clone(), kp, vp, out))
    assert int(ctx.status.item()) == 0
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,G,dk,dv,rot,turned", [(3, 1, 64, 64, 64, True), (4, 2, 128, 48, 32, True),
                                                   (2, 2, 24, 8, 16, False), (8, 4, 256, 256, 256, True),
                                                   (1, 1, 24, 16, 0, False), (4, 4, 72, 40, 64, True)])
@pytest.mark.parametrize("write", [True, False])
def test_rotation_in_groups_of_eight(H, G, dk, dv, rot, turned, write):
    """bfloat16 rows of whole groups of eight, and where only groups of four fit: the same bits."""
    from distengine_b200.kernels import recurrent as rk
    lens, page, g = (5, 1, 9), 8, _gen(dk)
    ctx = _ctx(lens, (3, 900, 0), (1, 0, 2))
    n = sum(lens)
    proj = torch.randn(n, H * dk + G * (dk + dv), generator=g).to(torch.bfloat16)
    fk, fv = torch.rand(rot // 2, generator=g).to(DEV), torch.rand(dv // 2, generator=g).to(DEV)
    table = torch.full((3, 120), -1, dtype=torch.int32)
    table[1, 0], table[0, 112], table[2, 0], table[2, 1] = 2, 0, 3, 1
    results = []
    for pad in (8 - proj.shape[1] % 8, 12 - proj.shape[1] % 8):
        p = _rows(proj, pad)
        kp = torch.zeros(4, G, page, dk, dtype=torch.bfloat16, device=DEV)
        vp = torch.zeros(4, G, page, dv, dtype=torch.bfloat16, device=DEV)
        rk.kv_write_rotated(p, fk, rot, fv if turned else None, H, G, dk, dv, kp, vp, table.to(DEV),
                            write, ctx)
        results.append((p.clone(), kp, vp))
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [1, 2, 4, 5])
@pytest.mark.parametrize("biased", [True, False])
def test_taps_by_tap(dtype, K, biased):
    from distengine_b200.kernels import recurrent as rk
    H, G, dk, dv, page, g = 4, 2, 64, 64, 16, _gen(K)
    lens, C = (7, 1, 3), (H + G) * dk + G * dv
    ctx = _ctx(lens, (0, 20, 2), (1, 0, 2))
    n = sum(lens)
    taps, bias = torch.randn(C, K, generator=g), torch.randn(C, generator=g)
    state = torch.randn(3, max(K - 1, 1) * C, generator=g).to(DEV)
    table = torch.tensor([[-1, 3], [0, -1], [2, -1]], dtype=torch.int32, device=DEV)
    proj = torch.randn(n, C, generator=g).to(dtype)
    results = []
    for by_tap, pad in ((False, 8), (True, 8), (True, 3)):
        q = torch.empty(n, H * dk, dtype=dtype, device=DEV)
        kp = torch.zeros(4, G, page, dk, dtype=dtype, device=DEV)
        vp = torch.zeros(4, G, page, dv, dtype=dtype, device=DEV)
        rk.qkv_prepare(_rows(proj, pad), q, H, G, dk, dv, kp, vp, table, ctx,
                       bias=bias.to(DEV) if biased else None,
                       taps=(taps.t().contiguous() if by_tap else taps).to(DEV), by_tap=by_tap,
                       kept=(state, 0) if K > 1 else None)
        results.append((q, kp, vp))
    assert int(ctx.status.item()) == 0
    for other in results[1:]:
        for a, b in zip(results[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,dv,turned", [(16, 40, True), (10, 64, False), (5, 128, True), (4, 160, True),
                                         (159, 4, False)])
@pytest.mark.parametrize("gate", [None, "feature", "head"])
def test_finish_of_rows_of_640_features(dtype, H, dv, turned, gate):
    """Rows around the 640 features from which four are taken at a time."""
    from distengine_b200.kernels import recurrent as rk
    n, g = 9, _gen(dv)
    ctx = _ctx((5, 4), (3, 900), (1, 0))
    o = torch.randn(n, H * dv, generator=g).to(DEV)
    fv = torch.rand(dv // 2, generator=g).to(DEV) if turned else None
    gt = None if gate is None else torch.randn(n, H * dv if gate == "feature" else H, generator=g).to(dtype)
    results = []
    for shift in (0, 1):                                  # results at 16-byte addresses, or not
        out = torch.zeros(n * H * dv + 8, dtype=dtype, device=DEV)[shift: shift + n * H * dv].view(n, -1)
        rk.attention_finish(o, fv, None if gt is None else gt.to(DEV), out, H, dv, ctx,
                            **({"gate_per_head": True} if gate == "head" else {}))
        results.append(out.clone())
    assert torch.equal(*results)



@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,H,G,rot,adjacent,K,norm,magnitude,temp,from_keys", [
    (128, 5, 1, 128, True, 3, True, 1.0, None, False), (128, 3, 3, 128, False, 4, True, 1.25, (0.3, 64), False),
    (64, 6, 2, 64, False, 2, False, 1.0, None, False), (64, 5, 1, 32, False, 3, True, 1.0, (0.3, 16), True),
    (128, 16, 4, 24, False, None, True, 1.0, None, False), (64, 1, 1, 12, True, 4, "plain", 1.0, None, False),
    (128, 4, 2, 0, False, None, False, 1.0, (0.1, 8), True),
])
@pytest.mark.parametrize("lens,starts", [((128,), (0,)), ((61, 1, 2, 3, 70), (0, 40, 1, 2, 9)),
                                         ((801,), (5,))])
def test_preparation_in_runs_of_tokens(dtype, D, H, G, rot, adjacent, K, norm, magnitude, temp,
                                             from_keys, lens, starts):
    """128 tokens and more: against the kernel with a token a block, which rows at other addresses
    reach.  Portions that begin inside a run, and behind 0 to 3 kept rows."""
    from distengine_b200.kernels import recurrent as rk
    page, g = 16, _gen(D + H)
    slots = tuple(range(len(lens)))
    ctx = _ctx(lens, starts, slots)
    n, C = sum(lens), (H + (G if from_keys else 2 * G)) * D
    need = [(s + l + page - 1) // page for s, l in zip(starts, lens)]
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    order, at = torch.randperm(sum(need), generator=g).int(), 0
    for i, m in enumerate(need):
        table[i, :m] = order[at: at + m]
        at += m
    proj = torch.randn(n, C, generator=g).to(dtype)
    bias = torch.randn(C, generator=g).to(DEV) if K else None
    taps = torch.randn(K, C, generator=g).to(DEV) if K else None
    state = torch.randn(len(lens), 4 * C, generator=g).to(DEV)
    weights = [torch.rand(D, generator=g).to(DEV) + 0.5 for _ in range(2)] if norm is True else [None, None]
    freq = (torch.rand(rot // 2, generator=g) * 2).to(DEV)
    results = []
    for pad in (8, 7):
        q = torch.zeros(n, H * D, dtype=dtype, device=DEV)
        kp = torch.zeros(sum(need), G, page, D, dtype=dtype, device=DEV)
        vp = torch.zeros(sum(need), G, page, D, dtype=dtype, device=DEV)
        rk.qkv_prepare(_rows(proj, pad), q, H, G, D, D, kp, vp, table.to(DEV), ctx, bias=bias, taps=taps,
                       by_tap=True, kept=(state, 0) if K else None,
                       norm=("head", *weights, 1e-5) if norm else None,
                       rotation=(freq, magnitude, adjacent), temperature=temp, values_from_keys=from_keys)
        results.append((q, kp, vp))
    assert int(ctx.status.item()) == 0
    for a, b in zip(*results):
        assert torch.equal(a, b)
