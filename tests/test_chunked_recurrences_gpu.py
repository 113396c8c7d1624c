"""The recurrences in chunks of 64 tokens, and the kernels around them that take four channels at a
time, against 64-bit token-by-token loops."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

import plain_vomotar as pv
from test_vomotar_mechanisms_gpu import _ctx, _gen, _scan_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.0 ** -24


def _step(lens, slots):
    from distengine_b200.kernels import recurrent as rk
    from distengine_b200.parts.recurrent import ChunkedMixer
    ctx = _ctx(lens, [0] * len(lens), slots)
    arrays, notes = {}, {}
    prep = SimpleNamespace(host=ctx.host, notes=notes,
                           add=lambda name, a: arrays.__setitem__(name, torch.from_numpy(a).to(DEV)))
    ChunkedMixer.prepare(SimpleNamespace(), prep)
    ctx.buffer = lambda name, shape, dtype: torch.full(shape, float("nan"), dtype=dtype, device=DEV)
    longest = rk.CHUNKED_PORTION - 1 if notes["recurrent/chunks"] else 0
    return ctx, arrays.get("recurrent/items"), arrays.get("recurrent/portions"), longest


# bound: the sums over a chunk (64 terms, or dk) and over the chunks that a decay leaves, each term
# of the size of the largest result, in float32: 64 + 128 roundings of 2^-24, doubled
BOUND = 2 * (64 + 128) * EPS


@pytest.mark.parametrize("rule", ["delta", "decay", "decay-bf16"])
@pytest.mark.parametrize("dk,dv,rep", [(64, 64, 1), (64, 192, 2), (128, 128, 2)])
@pytest.mark.parametrize("fast", [False, True])
def test_recurrences_in_chunks(rule, dk, dv, rep, fast):
    """Portions of whole chunks, of one token and one token less in the last, short ones between
    them that go token by token; states carried on; decays near 1 and down to 1e-8 a token."""
    from distengine_b200.kernels import recurrent as rk
    H, lens, slots = 4, (257, 7, 192, 255), (3, 0, 4, 1)
    assert rk.CHUNKED_PORTION == 192
    ctx, items, portions, longest = _step(lens, slots)
    n, g = sum(lens), _gen(dk + dv)
    state = torch.randn(6, H * dk * dv + 12, generator=g) * 0.3
    old = state.clone()
    state = state.to(DEV)
    out = torch.full((n, H * dv), float("nan"), device=DEV)
    flat = lambda t: t.reshape(n, -1).to(DEV).contiguous()
    if rule == "delta":
        G = H // rep
        q, k, v, beta, dec = _scan_inputs(n, H, G, dk, dv, 5)
        if fast:
            dec = dec ** torch.logspace(-3, 2, dk)
        rk.delta_chunks(flat(q), flat(k), flat(v), state, out, H, G, dk, dv, flat(dec), flat(beta),
                        items, portions, ctx)
        rk.state_scan(flat(q), flat(k), flat(v), state, out, H, G, dk, dv, ctx, g=flat(dec),
                      beta=flat(beta), longest=longest)
        q, k = q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1)
        dec = dec.double()
    else:
        q, k, v = (torch.randn(n, H, d, generator=g) * s for d, s in ((dk, dk ** -0.5), (dk, 0.3),
                                                                      (dv, 1.0)))
        v = v.to(torch.bfloat16 if rule == "decay-bf16" else torch.float32)
        decay = torch.tensor([1e-8, 0.3, 0.9, 1.0] if fast else [0.99, 0.999, 0.9, 0.97])
        for walk, extra in ((rk.decay_chunks, (decay.to(DEV), items, portions, ctx)),
                            (rk.state_scan, (ctx,))):
            heads = (H, H) if walk is rk.state_scan else (H,)
            more = dict(decay=decay.to(DEV), longest=longest) if walk is rk.state_scan else {}
            walk(flat(q), flat(k), flat(v), state, out, *heads, dk, dv, *extra, **more)
        dec, beta = decay.double()[None, :, None].expand(n, H, dk), None
    at = 0
    for i, m in enumerate(lens):
        S = old[slots[i], : H * dk * dv].double().view(H, dk, dv)
        want = torch.zeros(m, H, dv, dtype=torch.float64)
        for t in range(m):
            j = at + t
            S = S * dec[j][:, :, None]
            u = v[j].double()
            if beta is not None:
                u = beta[j].double()[:, None] * (u - torch.einsum("hkv,hk->hv", S, k[j].double()))
            S = S + k[j].double()[:, :, None] * u[:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", S, q[j].double())
        got = out[at: at + m].double().cpu().view(m, H, dv)
        err = (got - want).abs().max().item() / want.abs().max().item()
        assert err <= BOUND, (rule, i, err)
        end = state[slots[i], : H * dk * dv].double().cpu().view(H, dk, dv)
        err = (end - S).abs().max().item() / S.abs().max().item()
        assert err <= BOUND, (rule, "state", i, err)
        at += m
    untouched = [s for s in range(6) if s not in slots]
    assert torch.equal(state[untouched].cpu(), old[untouched])
    assert torch.equal(state[:, H * dk * dv:].cpu(), old[:, H * dk * dv:])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K,G,H,dk,dv,lens", [(1, 2, 2, 64, 64, (127, 1)), (2, 1, 3, 128, 128, (3, 130)),
                                              (3, 4, 4, 64, 96, (9, 2, 140)), (4, 2, 4, 128, 64, (1, 2, 3, 129)),
                                              (4, 2, 2, 64, 64, (127,))])
def test_delta_preparation_in_runs(dtype, K, G, H, dk, dv, lens):
    """Sequences that start within a run of eight tokens, fresh ones beside one whose earlier inputs
    come from its state, steps around the 128 tokens from which runs are taken."""
    from distengine_b200.kernels import recurrent as rk
    g, n, C = _gen(K), sum(lens), 2 * G * dk + H * dv
    proj = torch.randn(n, C + 4 + H + 4, generator=g)[:, : C + 4 + H + (-H) % 4].to(dtype).contiguous()
    a = torch.randn(n, H * dk, generator=g)
    taps, dt_bias = torch.randn(C, K, generator=g), torch.randn(H * dk, generator=g)
    a_log = torch.randn(H, generator=g) * 0.5
    rows = H * dk * dv
    state = torch.randn(len(lens) + 1, rows + (K - 1) * C, generator=g).to(dtype).float()
    pos0 = [0] * len(lens)
    pos0[-1] = 50                                         # the last one has gone before
    slots = list(range(len(lens), 0, -1))
    state[slots[:-1], rows:] = 0.0                        # as a slot is handed out
    ctx = _ctx(lens, pos0, slots)
    bufs = [torch.full((n, w), float("nan"), device=DEV)
            for w in (G * dk, G * dk, H * dv, H, H * dk)]
    rk.delta_prep(proj.to(DEV), a.to(DEV), taps.to(DEV), dt_bias.to(DEV), a_log.to(DEV),
                  state.to(DEV), rows, ctx, *bufs, H, G, dk, dv, C + 4)
    y, at = [], 0
    for i, m in enumerate(lens):
        before = state[slots[i], rows:].double().view(K - 1, C)
        x = torch.cat((before, proj[at: at + m, :C].double()))
        y.append(pv.silu(pv.causal_conv(x, taps.double()))[K - 1:])
        at += m
    y = torch.cat(y)
    want = [pv.unit(y[:, : G * dk].view(n, G, dk)) * dk ** -0.5,
            pv.unit(y[:, G * dk: 2 * G * dk].view(n, G, dk)), y[:, 2 * G * dk:],
            torch.sigmoid(proj[:, C + 4: C + 4 + H].double()),
            torch.exp(-torch.exp(a_log.double())[None, :, None]
                      * pv.softplus(a.double() + dt_bias.double()).view(n, H, dk))]
    for got, ref, name in zip(bufs, want, ("q", "k", "v", "beta", "decay")):
        ref = ref.reshape(n, -1)
        err = (got.double().cpu() - ref).abs().max().item()
        # float32: up to K products, a sum of dk squares, a few functions of 2 to 4 units each; the
        # decay's exponent may be a few tens
        assert err <= 64 * EPS * max(1.0, ref.abs().max().item()), (name, err)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,cols,pad", [(1, 4, 0), (3, 1028, 4), (5, 516, 8), (130, 2048, 0), (7, 258, 2),
                                        (3, 4096, 4)])
def test_rows_in_groups_of_four(dtype, n, cols, pad):
    from distengine_b200.kernels import recurrent as rk
    g = _gen(cols)
    x = (torch.randn(n, cols + pad, generator=g) * 4).to(dtype)
    o, w = torch.randn(n, cols, generator=g), torch.rand(cols, generator=g) + 0.5
    wide = x.to(DEV)
    out = torch.full((n, cols), float("nan"), device=DEV)
    rk.silu_rows(wide[:, pad:], out)
    want = pv.silu(x[:, pad:].double())
    assert (out.double().cpu() - want).abs().max().item() <= 8 * EPS * want.abs().max().item()
    res = torch.empty(n, cols, dtype=dtype, device=DEV)
    rk.head_gate(o.to(DEV), wide[:, pad:], w.to(DEV), res, 1, cols, 1e-5, spanning=True)
    o = o.double()
    want = (o / torch.sqrt((o * o).mean(1, keepdim=True) + 1e-5) * w.double()
            * torch.sigmoid(x[:, pad:].double()))
    unit = 16 * EPS if dtype == torch.float32 else 2.0 ** -8 + 16 * EPS
    assert ((res.double().cpu() - want).abs() <= unit * want.abs() + 1e-7).all()


@pytest.mark.parametrize("K,G,H,dk,dv", [(4, 2, 4, 64, 64), (2, 1, 2, 128, 192), (3, 4, 4, 128, 64),
                                         (1, 2, 2, 64, 320)])
def test_delta_preparation_of_any_number_of_tokens(K, G, H, dk, dv):
    """In float32 a token's vectors are the same bits in a step of 840 tokens of three sequences, which
    is prepared in runs, and in steps of fewer than 128 tokens of one, which are not."""
    from distengine_b200.kernels import recurrent as rk
    lens, pos0, C, g = (501, 3, 336), (0, 50, 7), 2 * G * dk + H * dv, _gen(dk)
    n, rows = sum(lens), H * dk * dv
    proj, a = torch.randn(n, C + H, generator=g).to(DEV), torch.randn(n, H * dk, generator=g).to(DEV)
    rest = [t.to(DEV) for t in (torch.randn(C, K, generator=g), torch.randn(H * dk, generator=g),
                                torch.randn(H, generator=g) * 0.5)]
    kept = torch.randn(3, rows + (K - 1) * C, generator=g).to(DEV)

    def prepare(lens, pos0, slots, first, state):
        m = sum(lens)
        bufs = [torch.full((m, w), float("nan"), device=DEV)
                for w in (G * dk, G * dk, H * dv, H, H * dk)]
        rk.delta_prep(proj[first: first + m], a[first: first + m], *rest, state, rows,
                      _ctx(lens, pos0, slots), *bufs, H, G, dk, dv, C)
        return bufs

    together = prepare(lens, pos0, (0, 1, 2), 0, kept)
    parts, first = [], 0
    for slot, length in enumerate(lens):
        state, at = kept.clone(), 0
        while at < length:
            m = min(127, length - at)
            parts.append(prepare([m], [pos0[slot] + at], [slot], first, state))
            if K > 1:
                state[slot, rows:] = torch.cat((state[slot, rows:].view(K - 1, C), proj[
                    first: first + m, :C]))[-(K - 1):].reshape(-1)
            at, first = at + m, first + m
    for got, want, name in zip(together, (torch.cat(x) for x in zip(*parts)),
                               ("q", "k", "v", "beta", "decay")):
        assert torch.equal(got, want), name


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,cols", [(157, 4100), (300, 2000), (1201, 516), (300, 1996)])
def test_silu_of_many_rows(dtype, n, cols):
    """Around the 600,000 elements from which a thread takes four groups of four, remainders of a grid's
    last round among them."""
    from distengine_b200.kernels import recurrent as rk
    x = (torch.randn(n, cols + 4, generator=_gen(n)) * 4).to(dtype)
    out = torch.full((n, cols), float("nan"), device=DEV)
    rk.silu_rows(x.to(DEV)[:, 4:], out)
    want = pv.silu(x[:, 4:].double())
    assert (out.double().cpu() - want).abs().max().item() <= 8 * EPS * want.abs().max().item()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,cols", [(97, 4100), (100, 4000), (781, 516), (3, 140004)])
def test_silu_of_rows_by_fours(dtype, n, cols):
    """Around the 400,000 elements from which a thread takes a group of four of four rows, remainders of
    four rows and of 1,024 columns among them."""
    test_silu_of_many_rows(dtype, n, cols)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,cols", [(6251, 64), (100003, 4), (4001, 100), (1563, 256), (397, 1012), (394, 1020)])
def test_silu_of_narrow_rows(dtype, n, cols):
    """Fewer than 1,024 columns: a block takes as many fours of rows as it has threads for."""
    test_silu_of_many_rows(dtype, n, cols)


def _walk(rule, lens, inputs, state, H, dk, dv, begin=0):
    """The tokens from ``begin`` on of one sequence, in steps of ``lens``: portions of 192 tokens and
    more by chunks, others by the scan.  Returns the read-outs."""
    from distengine_b200.kernels import recurrent as rk
    q, k, v, beta, dec = inputs
    outs = []
    for n in lens:
        ctx, items, portions, longest = _step([n], [0])
        flat = lambda t: t[begin: begin + n].reshape(n, -1).to(DEV).contiguous()
        out = torch.full((n, H * dv), float("nan"), device=DEV)
        if rule == "delta" and longest:
            rk.delta_chunks(flat(q), flat(k), flat(v), state, out, H, H, dk, dv, flat(dec), flat(beta),
                            items, portions, ctx)
        elif rule == "delta":
            rk.state_scan(flat(q), flat(k), flat(v), state, out, H, H, dk, dv, ctx, g=flat(dec),
                          beta=flat(beta))
        elif longest:
            rk.decay_chunks(flat(q), flat(k), flat(v), state, out, H, dk, dv, dec, items, portions, ctx)
        else:
            rk.state_scan(flat(q), flat(k), flat(v), state, out, H, H, dk, dv, ctx, decay=dec)
        outs.append(out)
        begin += n
    return torch.cat(outs)


@pytest.mark.parametrize("rule", ["delta", "decay"])
@pytest.mark.parametrize("dim", [64, 128])
def test_cuts_on_both_sides_of_the_line(rule, dim):
    """One prompt whole, in portions that the scan takes and in portions of both kinds: the same but
    for the order of float32 sums, each within the bound of the test above."""
    H, n = 2, 460
    inputs = list(_scan_inputs(n, H, H, dim, dim, 9))
    if rule == "decay":
        inputs[4] = torch.tensor([0.99, 0.97]).to(DEV)
    results = []
    for lens in ((460,), (150, 150, 160), (200, 60, 200), (191, 192, 77)):
        state = torch.zeros(1, H * dim * dim, device=DEV)
        out = _walk(rule, lens, inputs, state, H, dim, dim)
        results.append((out.double(), state.double()))
    for out, state in results[1:]:
        for got, want in ((out, results[0][0]), (state, results[0][1])):
            assert (got - want).abs().max().item() <= 2 * BOUND * want.abs().max().item()


def _layer(kind, dtype, taps=3):
    from distengine_b200.config.model import PartSpec
    from distengine_b200.parts import build_mixer
    width, heads, dim = 64, 2, 64
    params = dict(width=width, heads=heads, key_dim=dim, value_dim=dim, eps=1e-5)
    if kind == "gated_delta_rule":
        params.update(kv_heads=heads, taps=taps, rank=8)
    else:
        params.update(decay=(0.99, 0.97))
        if kind == "retention":
            params.update(rotary_dim=dim, theta=1e4)
    mixer = build_mixer(PartSpec.of(kind, **params), dtype, torch.device(DEV))
    g = _gen(4)
    mixer.load({name: (torch.randn(*shape, generator=g) * (0.1 if role == "matrix" else 0.3)).to(
        dtype if role == "matrix" else torch.float32) for name, (shape, role) in mixer.tensors().items()})
    return mixer, width


def _feed(mixer, x, dtype, lens):
    """One sequence through a layer in steps of ``lens``; its outputs and the state it leaves."""
    from gpu_helpers import PartHarness
    harness = PartHarness([mixer], [mixer.cache_spec()], dtype, max_seqs=2)
    outs, at = [], 0
    for n in lens:
        outs.append(harness.run([("a", n)], lambda ctx, bindings: mixer.forward(
            x[at: at + n], ctx, bindings[0]).clone()))
        at += n
    return torch.cat(outs), harness.cache.bindings()[0].state[harness.cache.slot("a")].clone()


@pytest.mark.parametrize("kind", ["gated_delta_rule", "retention", "lightning_attention"])
def test_a_float32_layer_does_not_depend_on_the_cut(kind):
    """In float32 a prompt's results and the state it leaves are the same bits however it was cut,
    portions of 192 tokens and more among them."""
    mixer, width = _layer(kind, torch.float32)
    x = torch.randn(900, width, generator=_gen(8)).to(DEV)
    out, state = _feed(mixer, x, torch.float32, (900,))
    for lens in ((191, 192, 517), (1, 640, 259), (100,) * 9):
        other, end = _feed(mixer, x, torch.float32, lens)
        assert torch.equal(other, out) and torch.equal(end, state), lens


@pytest.mark.parametrize("rule", ["delta", "decay"])
@pytest.mark.parametrize("group", [1, 2, 5])
def test_chunks_a_few_at_a_time(rule, group, monkeypatch):
    """A workspace of a few chunks, smaller than the step and cutting its portions: the same bits as
    all at once, and no buffer is larger."""
    from distengine_b200.kernels import recurrent as rk
    H, dk, dv, lens, slots = 2, 64, 128, (257, 193, 320), (2, 0, 1)
    n, g = sum(lens), _gen(group)
    q, k, v, beta, dec = _scan_inputs(n, H, H, dk, dv, 5)
    flat = lambda t: t.reshape(n, -1).to(DEV).contiguous()
    start = torch.randn(3, H * dk * dv, generator=g).to(DEV)
    a_chunk = H * (2 * 64 * 64 + 4 * dk * 64 + dk + 64 * dv + dk * dv if rule == "delta"
                   else dk * 64 + 64 * 64 + dk * dv)
    results = []
    for work in (1 << 26, group * a_chunk + a_chunk // 2):
        monkeypatch.setattr(rk, "CHUNK_WORK", work)
        ctx, items, portions, _ = _step(lens, slots)
        assert items.shape[0] == 14
        make, sizes = ctx.buffer, []
        ctx.buffer = lambda name, shape, dtype: (sizes.append(shape[0]), make(name, shape, dtype))[1]
        state, out = start.clone(), torch.full((n, H * dv), float("nan"), device=DEV)
        if rule == "delta":
            rk.delta_chunks(flat(q), flat(k), flat(v), state, out, H, H, dk, dv, flat(dec), flat(beta),
                            items, portions, ctx)
        else:
            rk.decay_chunks(flat(q), flat(k), flat(v), state, out, H, dk, dv,
                            torch.tensor([0.99, 0.9]).to(DEV), items, portions, ctx)
        assert len(sizes) == 1 and min(14, work // a_chunk) * a_chunk <= sizes[0] <= work
        results.append((out, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("kind,taps", [("gated_delta_rule", 3), ("gated_delta_rule", 1),
                                       ("retention", 0), ("lightning_attention", 0)])
def test_steps_by_chunks_as_graphs(kind, taps):
    """A bfloat16 step of a long portion beside a short one, or alone (with one tap the scan then has
    nothing to do), replayed as a CUDA graph: the bits of the step launch by launch."""
    from gpu_helpers import PartHarness
    from distengine_b200.kernels import recurrent as rk
    mixer, width = _layer(kind, torch.bfloat16, taps or 3)
    for lens in ((900, 37), (900,)):
        assert rk.chunks_pay(kind == "gated_delta_rule", 2, 64, 64, 900, 900, 15)
        harness = PartHarness([mixer], [mixer.cache_spec()], torch.bfloat16, num_pages=80, max_seqs=2,
                              max_len=2048)
        harness.runner.use_graphs = True
        x = torch.randn(sum(lens), width, generator=_gen(8)).to(torch.bfloat16).to(DEV)
        names, results = [f"r{i}" for i in range(len(lens))], []
        for _ in range(7):
            out = harness.run(list(zip(names, lens)),
                              lambda ctx, bindings: mixer.forward(x, ctx, bindings[0]))
            states = [harness.cache.bindings()[0].state[harness.cache.slot(n)].clone() for n in names]
            results.append((out.clone(), torch.stack(states)))
            for name in names:
                harness.cache.release(name)
        assert harness.runner.graph_replays >= 2
        for out, state in results[1:]:
            assert torch.equal(out, results[0][0]) and torch.equal(state, results[0][1])


@pytest.mark.parametrize("kind,taps", [("gated_delta_rule", 3), ("gated_delta_rule", 1),
                                       ("lightning_attention", 0)])
def test_a_bfloat16_layer_by_chunks_and_by_the_scan(kind, taps, monkeypatch):
    """The same step both ways: the states within the bound of float32 sums, the outputs within two
    roundings of bfloat16; and portions that are not in whole 16-byte pieces go by the scan."""
    from distengine_b200.kernels import recurrent as rk
    mixer, width = _layer(kind, torch.bfloat16, taps or 3)
    x = torch.randn(900, width, generator=_gen(8)).to(torch.bfloat16).to(DEV)
    out, state = _feed(mixer, x, torch.bfloat16, (900,))
    monkeypatch.setattr(rk, "chunks_pay", lambda *a: False)
    other, end = _feed(mixer, x, torch.bfloat16, (900,))
    assert not torch.equal(end, state)                       # (two ways)
    assert (end - state).abs().max().item() <= 2 * BOUND * state.abs().max().item()
    assert (other.float() - out.float()).abs().max().item() <= 2 ** -6 * out.float().abs().max().item()
    monkeypatch.undo()
    monkeypatch.setattr(rk, "chunks_aligned", lambda v, state: False)
    last, end_too = _feed(mixer, x, torch.bfloat16, (900,))
    assert torch.equal(last, other) and torch.equal(end_too, end)
