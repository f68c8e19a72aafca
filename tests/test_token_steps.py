"""Kernels of steps of few tokens that do several parts' work in one launch, at the edges of their sizes."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from janus_b200.kernels import ops
    return ops


def rnd(g, *shape, s=1.0):
    return (torch.randn(*shape, generator=g, dtype=torch.float64) * s).float()


def plain_step(kind, x, raw, S, n, m, H, G, d, e, cols, p0, p1, scalar, rank):
    """One token of one sequence in float64: (heads' outputs [H, e], S, n, m)."""
    q_col, k_col, v_col, a_col, b_col = cols
    x, raw, S, p0, p1 = x.double(), raw.double(), S.double(), p0.double(), p1.double()
    q, k = (x[c: c + G * d].view(G, d).repeat_interleave(H // G, 0) for c in (q_col, k_col))
    v = x[v_col: v_col + H * e].view(H, e)
    if kind == "delta":
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + scalar) * d ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + scalar)
        beta = torch.sigmoid(raw[a_col: a_col + H])[:, None]
        S = S * torch.exp(-torch.exp(p0) * F.softplus(raw[b_col: b_col + H] + p1))[:, None, None]
        S = S + k[:, :, None] * (beta * (v - torch.einsum("hde,hd->he", S, k)))[:, None, :]
        return torch.einsum("hde,hd->he", S, q), S, n, m
    q = q * d ** -0.5
    if kind == "channel":
        z = p1 + raw[a_col: a_col + rank] @ p0
        S = S * torch.exp(F.logsigmoid(z) * scalar).view(H, d, 1) + k[:, :, None] * v[:, None, :]
        return torch.einsum("hde,hd->he", S, q), S, n, m
    gi = scalar * torch.tanh((raw[a_col: a_col + H] + p0) / scalar)
    gf = F.logsigmoid(scalar * torch.tanh((raw[b_col: b_col + H] + p1) / scalar))
    m, n = m.double(), n.double()
    new = torch.maximum(gf + m, gi)
    keep, take = torch.exp(gf + m - new), torch.exp(gi - new)
    S = keep[:, None, None] * S + take[:, None, None] * k[:, :, None] * v[:, None, :]
    n = keep[:, None] * n + take[:, None] * k
    below = torch.maximum((n * q).sum(-1).abs(), torch.exp(-new)) + 1e-6
    return torch.einsum("hde,hd->he", S, q) / below[:, None], S, n, new


@pytest.mark.parametrize("kind", ["delta", "memory", "channel"])
@pytest.mark.parametrize("T, H, G, d, e", [(1, 2, 1, 128, 128), (3, 4, 2, 64, 64), (2, 1, 1, 4, 4), (5, 3, 3, 100, 68),
                                           (2, 2, 2, 128, 256), (1, 6, 2, 36, 132), (70, 2, 1, 8, 60)])
def test_head_step(ops, kind, T, H, G, d, e):
    """A token of every sequence against the formulas in float64.  Sums of at most 128 products and the norm of e numbers, each
    rounded to half of 2^-23, and a few exponentials of some ulps: 1e-5 of the largest result leaves a factor of ten."""
    if kind != "delta":
        G = H
    g = torch.Generator().manual_seed(T * 1000 + d + e)
    rank, gap = 12 if d < 100 else 65, 4
    q_col, k_col = gap, gap + G * d
    v_col = k_col + G * d
    a_col = v_col + H * e
    b_col = a_col + H
    gate_col = max(b_col + H, a_col + rank)
    rows = rnd(g, T, gate_col + H * e + 3)
    rows[:, a_col:gate_col] *= 2.0
    p0 = rnd(g, rank, H * d, s=0.3) if kind == "channel" else rnd(g, H, s=0.5)
    p1 = rnd(g, H * d) if kind == "channel" else rnd(g, H)
    scalar = {"delta": 1e-6, "memory": 3.0, "channel": 1.0 / 16}[kind]
    weight = rnd(g, H * e) if kind == "memory" else rnd(g, e)
    ex = e + (kind == "memory")
    m_off = H * d * ex
    state = rnd(g, T + 2, (m_off + H + 3) // 4 * 4)
    slots = torch.randperm(T + 2, generator=g)[:T].int()
    for dtype in (torch.float32, torch.bfloat16):
        got_state, out = state.to(DEV), torch.full((T, H * e), float("nan"), dtype=dtype, device=DEV)
        dev = rows.to(DEV)
        assert ops.head_step_supported(d, e, got_state, kind == "memory") == (d * ex % 4 == 0)
        if d * ex % 4:
            return
        ops.head_step(kind, dev, q_col, k_col, v_col, d ** -0.5, dev, a_col, b_col, p0.to(DEV), p1.to(DEV), scalar, got_state,
                      dev[:, gate_col: gate_col + H * e], weight.to(DEV), 1e-5, out, torch.arange(T + 1, dtype=torch.int32).to(DEV),
                      slots.to(DEV), H, G, d, e, m_off=m_off, sigmoid=kind == "memory")
        want_state = state.double().clone()
        for t in range(T):
            row = state[slots[t]]
            blocks = row[:m_off].view(H, d * ex)
            S, n, m = blocks[:, :d * e].reshape(H, d, e), blocks[:, d * e:], row[m_off: m_off + H]
            o, S, n, m = plain_step(kind, rows[t], rows[t], S, n, m, H, G, d, e, (q_col, k_col, v_col, a_col, b_col), p0, p1,
                                    scalar, rank)
            z = rows[t, gate_col: gate_col + H * e].double().view(H, e)
            y = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * weight.double().view(-1, e)
            y = y * (torch.sigmoid(z) if kind == "memory" else F.silu(z))
            err = (out[t].double().cpu().view(H, e) - y).abs().max() / y.abs().max()
            assert float(err) < (1e-5 if dtype == torch.float32 else 2.0 ** -8), (t, float(err))
            w = want_state[slots[t]]
            w[:m_off] = torch.cat([S.reshape(H, -1), n.double()], 1).reshape(-1) if kind == "memory" else S.reshape(-1)
            if kind == "memory":
                w[m_off: m_off + H] = m
        err = (got_state.double().cpu() - want_state).abs().max() / want_state.abs().max()
        assert float(err) < 1e-6, float(err)
        untouched = [s for s in range(T + 2) if s not in slots.tolist()]
        assert torch.equal(got_state[untouched].cpu(), state[untouched])


@pytest.mark.parametrize("T", [1, 5, 130])
@pytest.mark.parametrize("W, E, extra, top, softmax, groups, keep", [(2048, 8, 0, 2, False, 0, 0), (264, 8, 1, 2, True, 4, 2), (8, 3, 1, 3, False, 0, 0),
                                                                     (4096, 16, 0, 4, True, 0, 0), (1024, 40, 1, 6, False, 8, 3),
                                                                     (16, 4095, 1, 2, False, 0, 0)])
def test_route_tokens(ops, T, W, E, extra, top, softmax, groups, keep):
    """The router's product and choice in one launch: logits against float64 (each half of a row is lanes' chains of at most
    64 products and eight more sums: 72 roundings of 2^-24 of the sum of the products' sizes), the choice as `route_topk`
    makes it from the same logits, and a token's row whatever the number of tokens."""
    g = torch.Generator().manual_seed(W + E)
    x, w = rnd(g, T, W).bfloat16().to(DEV), rnd(g, E + extra, W).bfloat16().to(DEV)
    corr = rnd(g, E).to(DEV) if groups == 0 else None
    logits = torch.full((T, E + extra), float("nan"), device=DEV)
    sel_e, sel_w = torch.full((T, top), -1, dtype=torch.int32, device=DEV), torch.full((T, top), float("nan"), device=DEV)
    how = dict(softmax=softmax, groups=groups, keep=keep, experts=E, correction=corr, scale=1.5, shares=True)
    ops.route_tokens(x, w, logits, top, sel_e, sel_w, **how)
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((logits.double() - ref).abs() <= 72 * 2.0 ** -24 * size).all())
    e2, w2 = torch.empty_like(sel_e), torch.empty_like(sel_w)
    ops.route_topk(logits, top, e2, w2, **how)
    assert torch.equal(sel_e, e2) and torch.equal(sel_w, w2)
    one = torch.empty(1, E + extra, device=DEV)
    ops.route_tokens(x[T // 2: T // 2 + 1].contiguous(), w, one, top, e2[:1], w2[:1], **how)
    assert torch.equal(one[0], logits[T // 2]) and torch.equal(e2[0], sel_e[T // 2])


def plain_experts(x, sel_e, sel_w, wg, wu, wd, base, on_output):
    out = base.double().clone()
    x, wg, wu, wd = x.double(), wg.double(), wu.double(), wd.double()
    for t in range(x.shape[0]):
        for k in range(sel_e.shape[1]):
            e, s = int(sel_e[t, k]), float(sel_w[t, k])
            h = x[t] if on_output else x[t] * s
            a = (F.silu(wg[e] @ h) * (wu[e] @ h)).bfloat16().double()
            out[t] += (wd[e] @ a) * (s if on_output else 1.0)
    return out


@pytest.mark.parametrize("T, top, E, W, Fi, on_output", [(1, 2, 8, 256, 384, False), (1, 1, 1, 128, 128, True), (5, 3, 4, 384, 256, True),
                                                         (16, 2, 5, 128, 640, False), (17, 2, 40, 256, 128, True),
                                                         (33, 4, 3 + 4, 128, 256, False), (64, 2, 64, 128, 128, True),
                                                         (64, 8, 120, 128, 128, False), (2, 2, 8, 2048, 1024, True)])
def test_experts_stream(ops, T, top, E, W, Fi, on_output):
    """The streamed experts against float64 (their activations rounded to bfloat16, as the kernel's are), with slices of k
    that begin and end anywhere, experts nobody chose, one that all chose, and tokens on both sides of a tile.  An activation
    may round the other way (2^-8 of itself, in few of them): 2^-8 of the largest result bounds what that does to a sum."""
    g = torch.Generator().manual_seed(T * 100 + E)
    x = rnd(g, T, W).bfloat16()
    wg, wu, wd = (rnd(g, E, *s, s=W ** -0.5).bfloat16() for s in ((Fi, W), (Fi, W), (W, Fi)))
    sel_e = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).int()
    sel_e[:, 0] = torch.where((sel_e == 0).any(1), sel_e[:, 0], torch.zeros(T, dtype=torch.int32))     # all choose expert 0
    sel_w = torch.rand(T, top, generator=g) + 0.1
    base = rnd(g, T, W)
    assert ops.experts_stream_supported(T, top, E)
    gu = ops.pack_gated(wg.reshape(E * Fi, W).to(DEV), wu.reshape(E * Fi, W).to(DEV))
    dn = ops.pack_weight(wd.reshape(E * W, Fi).to(DEV))
    z = torch.zeros(T * top, 2 * Fi, device=DEV)
    act = torch.full((min(E, T * top) * T, Fi), float("nan"), dtype=torch.bfloat16, device=DEV)
    out, places = base.to(DEV), torch.empty(T * top, dtype=torch.int32, device=DEV)
    ops.experts_stream(x.to(DEV), sel_e.to(DEV), sel_w.to(DEV), gu, dn, E, z, act, places, out, weight_on_output=on_output)
    ops.check_kernel_status(torch.device(DEV))
    used = torch.unique(sel_e).tolist()
    assert places.tolist() == [used.index(e) for e in sel_e.reshape(-1).tolist()]
    want = plain_experts(x, sel_e, sel_w, wg, wu, wd, base, on_output)
    err = float((out.double().cpu() - want).abs().max() / (want - base.double()).abs().max())
    assert err < 2.0 ** -8, err
    for t in range(T):                     # the sums themselves, in float32
        for k in range(top):
            e = int(sel_e[t, k])
            ref = torch.cat([wg[e].double() @ x[t].double(), wu[e].double() @ x[t].double()])
            assert float((z[t * top + k].double().cpu() - ref).abs().max()) < 1e-5 * float(ref.abs().max()) + 1e-6


def test_experts_stream_refuses(ops):
    assert not ops.experts_stream_supported(65, 2, 8) and not ops.experts_stream_supported(1, 2, 513)
    assert not ops.experts_stream_supported(64, 8, 200)             # 200 experts x 64 tokens
    ops.set_deterministic(True)
    try:
        assert not ops.experts_stream_supported(1, 2, 8)
    finally:
        ops.set_deterministic(False)


def test_clear_rows(ops):
    """A row of many matrices at once: sizes that are whole vectors and sizes that are not, more matrices than a launch takes."""
    sizes = [4, 1, 7, 4096, 5000, 2 ** 20] + [8 + i for i in range(14)]
    m = [torch.ones(3, n, device=DEV) for n in sizes] + [torch.ones(3, 2, 5, device=DEV)]
    ops.clear_rows(m, 1)
    for t in m:
        assert float(t[1].abs().sum()) == 0.0 and bool((t[0] == 1).all()) and bool((t[2] == 1).all())


@pytest.mark.parametrize("T, H, e", [(1, 3, 128), (5, 1, 4), (7, 16, 100), (33, 2, 128), (300, 5, 64), (700, 15, 128), (1311, 10, 100),
                                     (4097, 5, 64), (3277, 100, 4)])
@pytest.mark.parametrize("per_head, sigmoid, divided", [(False, False, False), (True, True, True)])
def test_head_norm_gate_in_vectors(ops, T, H, e, per_head, sigmoid, divided):
    """Heads in whole vectors against float64 and against the general form (a gate whose rows are off a 16-byte boundary)."""
    g = torch.Generator().manual_seed(T + e)
    o, wide, w = rnd(g, T, H * e), rnd(g, T, H * e + 4), rnd(g, H * e if per_head else e)
    den = rnd(g, T, H).abs() + 0.5 if divided else None
    odd = torch.zeros(T, H * e + 5)
    odd[:, 1: H * e + 1] = wide[:, :H * e]
    x = o.double().view(T, H, e) / (1.0 if den is None else den.double()[:, :, None])
    z = wide[:, :H * e].double().view(T, H, e)
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double().view(-1, e) * (torch.sigmoid(z) if sigmoid else F.silu(z))
    for dtype, tol in ((torch.float32, 1e-6), (torch.bfloat16, 2.0 ** -8)):
        outs = []
        for gate in (wide.to(DEV)[:, :H * e], odd.to(DEV)[:, 1: H * e + 1]):
            out = torch.full((T, H * e), float("nan"), dtype=dtype, device=DEV)
            ops.head_norm_gate(o.to(DEV), gate, w.to(DEV), 1e-5, out, H, e, sigmoid=sigmoid, denom=None if den is None else den.to(DEV))
            outs.append(out.double().cpu().view(T, H, e))
            assert float(((outs[-1] - want).abs() / (want.abs() + want.abs().mean())).max()) < tol


@pytest.mark.parametrize("pairs, E", [(1, 1), (7, 3), (1024, 8), (8192, 8), (8193, 70), (20000, 1024)])
def test_expert_plan_counts(ops, pairs, E):
    """Pairs sorted by expert and the tiles of both products, at the edges of what a thread keeps and of warps."""
    g = torch.Generator().manual_seed(pairs)
    sel = torch.randint(0, E, (pairs, 1), generator=g).int()
    Fi, W = 384, 512
    mg, md = ops.grouped_max_items(pairs, E, Fi, "swiglu"), ops.grouped_max_items(pairs, E, W, "store")
    order, where = (torch.full((pairs,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    tg, td = (torch.full((4 + 4 * n,), -1, dtype=torch.int32, device=DEV) for n in (mg, md))
    ops.expert_plan(sel.to(DEV), E, Fi, W, order, where, tg, td)
    o, wh, s = order.cpu().long(), where.cpu().long(), sel[:, 0].long()
    assert torch.equal(torch.sort(o).values, torch.arange(pairs)) and torch.equal(wh[o], torch.arange(pairs))
    assert bool((s[o][1:] >= s[o][:-1]).all())
    counts = torch.bincount(s, minlength=E)
    starts = torch.cumsum(counts, 0) - counts
    for table, per, rows in ((tg.cpu(), 128, Fi), (td.cpu(), 256, W)):
        want = [(int(starts[e]) + 256 * tt, int(starts[e] + counts[e]), e * rows + per * ft, per * ft)
                for e in range(E) for ft in range(rows // per) for tt in range((int(counts[e]) + 255) // 256)]
        assert int(table[0]) == len(want)
        assert table[4: 4 + 4 * len(want)].view(-1, 4).tolist() == [list(w) for w in want]


@pytest.mark.parametrize("T", [64, 65, 71, 137])
def test_conv_taps_off_their_vectors(ops, T):
    """A prompt's taps are read four to a load where they begin on 16 bytes, else one by one: the same numbers either way."""
    g = torch.Generator().manual_seed(T)
    H, G, d, e, page, rot = 2, 1, 16, 12, 16, 8
    C = (2 * H + 2 * G) * d + G * e
    proj, loose, state = rnd(g, T, C).to(DEV), rnd(g, 4 * C + 1).to(DEV), rnd(g, 1, 3, C).to(DEV)
    angles = rnd(g, T, rot // 2)
    table = torch.stack([angles.cos(), angles.sin()], dim=-1).contiguous().to(DEV)
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, seq = torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    pages = -(-T // page)
    results = []
    for w in (loose[1:].view(C, 4), loose[1:].clone().view(C, 4)):
        q = torch.empty(T, 2 * H * d, device=DEV)
        k_cache, v_cache = torch.zeros(pages, 2 * G, page, d, device=DEV), torch.zeros(pages, G, page, e, device=DEV)
        ops.conv_rope_cache(proj, w, 4, state, seq, ints(0, T), ints(0), pos, table, rot, q, pos, k_cache, v_cache, H, G, d, e, page)
        results.append((q, k_cache, v_cache))
    assert all(torch.equal(a, b) for a, b in zip(*results)) and results[0][0].abs().max() > 0


class Scratch:
    """A workspace whose buffers come filled with NaN, and what was asked for."""

    def __init__(self):
        self.asked = []

    def get(self, name, shape, dtype):
        self.asked.append(name)
        return torch.full(shape, float("nan"), dtype=dtype, device=DEV)


def channel_walk(q, k, v, a, lens, S):
    """The recurrence with a decay a channel in the numbers' own type: (outputs [T, H, e], states [n, H, d, e])."""
    out, states, at = [], [], 0
    for n, s in zip(lens, S):
        for t in range(at, at + n):
            s = a[t, :, :, None] * s + k[t, :, :, None] * v[t, :, None, :]
            out.append(torch.einsum("hde,hd->he", s, q[t]))
        states.append(s)
        at += n
    return torch.stack(out), torch.stack(states)


@pytest.mark.parametrize("H, d, e, lens", [(2, 128, 64, [64]), (3, 100, 68, [33, 1, 130]), (1, 4, 10, [31, 65, 32]), (2, 64, 128, [97, 200]),
                                           (16, 128, 128, [70] * 10), (5, 128, 65, [1] * 40 + [161])])
@pytest.mark.parametrize("decays", ["mild", "strong", "any"])
def test_channel_chunks(ops, monkeypatch, H, d, e, lens, decays):
    """Prompts by chunks of 32 tokens with a decay a key channel: parts of a chunk, several sequences, one block an SM and two,
    columns that are no pairs, decays that are zero or below it, and the scratch in slabs.  An output's error is at most a
    rounding for each factor on the way to it, of the sum of its terms' sizes."""
    g = torch.Generator().manual_seed(H * 1000 + d + e)
    T, n, col = sum(lens), len(lens), 8
    proj = rnd(g, T, col + H * (2 * d + e) + (-(2 * H * d + H * e)) % 4)
    a = torch.rand(T, H * d, generator=g)
    a = 1 - 0.05 * a if decays == "mild" else a
    if decays == "any":
        a = (a * 2 - 1) * (torch.rand(T, H * d, generator=g) > 0.02)
    before, scale = rnd(g, n + 1, H * d * e), d ** -0.5
    slots = torch.randperm(n + 1, generator=g)[:n]
    q_start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist())
    parts = [proj[:, col: col + H * d].view(T, H, d) * scale, proj[:, col + H * d: col + 2 * H * d].view(T, H, d),
             proj[:, col + 2 * H * d: col + 2 * H * d + H * e].view(T, H, e), a.view(T, H, d)]
    S = before[slots].view(n, H, d, e)
    want, states = channel_walk(*(x.double() for x in parts), lens, S.double())
    size, state_size = channel_walk(*(x.double().abs() for x in parts), lens, S.double().abs())
    monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: True)
    for most in (ops.STATE_SCRATCH_BYTES, 1):                           # all chunks at once, and one of every sequence after another
        monkeypatch.setattr(ops, "STATE_SCRATCH_BYTES", most)
        out, state, ws = torch.full((T, H * e), float("nan"), device=DEV), before.to(DEV), Scratch()
        ops.gated_linear_scan(proj.to(DEV), col, col + H * d, col + 2 * H * d, scale, a.to(DEV), out, state, q_start.int().to(DEV),
                              slots.int().to(DEV), n, H, d, e, max(lens), ws)
        assert ws.asked == ["state_chunks"]
        bound = (d + 2 * max(lens) + 40) * 2.0 ** -24
        assert ((out.cpu().double().view(T, H, e) - want).abs() <= bound * size + 1e-30).all()
        got = state.cpu()[slots].double().view(n, H, d, e)
        assert ((got - states).abs() <= bound * state_size + 1e-30).all()
        rest = [s for s in range(n + 1) if s not in slots.tolist()]
        assert torch.equal(state.cpu()[rest], before[rest])


@pytest.mark.parametrize("what", ["value", "decay", "key"])
def test_channel_chunks_that_are_not_finite(ops, monkeypatch, what):
    """A value, a decay or a key that is not finite shows from its token on, in its column or its head, and nowhere else, by
    chunks as by the walk."""
    g = torch.Generator().manual_seed(3)
    H, d, e, lens, bad = 2, 128, 64, [200, 70], 77
    T, per = sum(lens), 128 * 64
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    proj, before, a = rnd(g, T, H * (2 * d + e)).to(DEV), rnd(g, 2, H * per).to(DEV), torch.rand(T, H * d, generator=g).to(DEV)
    monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: True)
    for ws in (Scratch(), None):
        results = []
        for sick in (True, False):
            x, w, out, state = proj.clone(), a.clone(), torch.zeros(T, H * e, device=DEV), before.clone()
            if sick:
                if what == "value":
                    x[bad, 2 * H * d + 3] = float("inf")
                elif what == "key":
                    x[bad, H * d + 5] = float("inf")
                else:
                    w[bad, 5] = float("nan")
            ops.gated_linear_scan(x, 0, H * d, 2 * H * d, 1.0, w, out, state, ints(0, 200, T), ints(1, 0), 2, H, d, e, 200, ws)
            results.append((out.view(T, H, e), state.view(2, H, d, e)))
        (got, state), (clean, clean_state) = results
        columns = slice(3, 4) if what == "value" else slice(0, e)
        assert not torch.isfinite(got[bad:200, 0, columns]).any()
        got[bad:200, 0, columns] = clean[bad:200, 0, columns]
        assert torch.equal(got, clean)
        assert not torch.isfinite(state[1, 0, :, columns] if what == "value" else state[1, 0, 5]).any()
        assert torch.equal(state[0], clean_state[0]) and torch.equal(state[1, 1], clean_state[1, 1])


@pytest.mark.parametrize("dtype, W, Fi", [(torch.bfloat16, 256, 128), (torch.bfloat16, 96, 64), (torch.bfloat16, 40, 24), (torch.float32, 64, 48)])
@pytest.mark.parametrize("T, top, on_output", [(1, 2, False), (5, 1, False), (16, 4, True), (40, 3, False)])
def test_deterministic_experts_are_added_in_order(ops, dtype, W, Fi, T, top, on_output):
    """Deterministic mode: a token's experts are added up in the order of its choices and the sum goes to the residual, whatever
    finishes first, so every run gives the same bits; and they are the bits of the experts' own results in that order."""
    from types import SimpleNamespace

    from janus_b200.engine.workspace import Workspace
    from janus_b200.parts.routed import RoutedExperts
    g, E = torch.Generator().manual_seed(T + W), 8
    ops.set_deterministic(True)
    try:
        part = RoutedExperts(W, Fi, E, top, weight_on="output" if on_output else "input", dtype=dtype,
                             device=torch.device(DEV))
        wts = {n: rnd(g, *s[0], s=s[0][-1] ** -0.5).to(dtype) for n, s in part.weight_shapes().items()}
        part.load(**wts)
        x, base = rnd(g, T, W).to(dtype).to(DEV), rnd(g, T, W).to(DEV)
        ctx = SimpleNamespace(is_decode=True, workspace=Workspace(torch.device(DEV)))

        def run(p):
            out = base.clone()
            p.forward(x, out, ctx)
            return out

        first = run(part)
        for _ in range(50):
            assert torch.equal(run(part), first)
        sel_e, sel_w = (ctx.workspace.get(n, (T, top), t).clone() for n, t in (("router_experts", torch.int32), ("router_weights", torch.float32)))
        sums = torch.zeros(T, W, device=DEV)
        for k in range(top):                     # the experts' results one by one, into zeros
            one, e, s = torch.zeros(T, W, device=DEV), sel_e[:, k:k + 1].contiguous(), sel_w[:, k:k + 1].contiguous()
            if dtype == torch.bfloat16 and W % 32 == 0 and Fi % 32 == 0:
                ops.experts_few_tokens_tc(x, e, s, part.w_gate, part.w_up, part.w_down, torch.empty(T, Fi, dtype=dtype, device=DEV), one,
                                          weight_on_output=on_output)
            else:
                ops.experts_few_tokens(x, e, s, part.w_gate, part.w_up, part.w_down, torch.empty(T, Fi, device=DEV), one,
                                       weight_on_output=on_output)
            sums += one
        assert torch.equal(first, base + sums)
    finally:
        ops.set_deterministic(False)


@pytest.mark.parametrize("tiles", [True, False])
@pytest.mark.parametrize("T, E, top, on_output", [(1, 8, 2, False), (17, 5, 1, True), (64, 40, 3, False)])
def test_routed_part_by_tiles_and_by_rows(ops, monkeypatch, tiles, T, E, top, on_output):
    """The whole part in a step of few tokens, in either form, with scratch that comes filled with NaN and with scratch that the
    launch before has cleared, against float64 (bound as in `test_experts_stream`; an input's weight is rounded with it by rows,
    2^-9 of a sum's terms more)."""
    from types import SimpleNamespace

    from janus_b200.engine.workspace import Workspace
    from janus_b200.parts.routed import RoutedExperts
    g, W, Fi = torch.Generator().manual_seed(T + E), 256, 128
    monkeypatch.setattr(ops, "experts_stream_pays", lambda *_: tiles)
    part = RoutedExperts(W, Fi, E, top, weight_on="output" if on_output else "input", device=torch.device(DEV))
    wts = {n: rnd(g, *s[0], s=s[0][-1] ** -0.5).bfloat16() for n, s in part.weight_shapes().items()}
    part.load(**wts)
    x, base = rnd(g, T, W).bfloat16(), rnd(g, T, W)
    ws = Workspace(torch.device(DEV))
    ctx = SimpleNamespace(is_decode=True, workspace=ws)
    for cleared in (False, True, True):
        out = base.to(DEV)
        scratch = part.scratch_to_clear(ctx, T)
        assert not tiles or tuple(scratch.shape) == (T * top, 2 * Fi)
        for buf in ws._buffers.values():
            if buf.is_floating_point():
                buf.fill_(float("nan"))
        if cleared and scratch is not None:
            scratch.zero_()
        part.forward(x.to(DEV), out, ctx, scratch_cleared=cleared)
        ops.check_kernel_status(torch.device(DEV))
        sel_e, sel_w = (ws.get(n, (T, top), t).cpu() for n, t in (("router_experts", torch.int32), ("router_weights", torch.float32)))
        wg, wu, wd = (torch.stack([wts[f"e{e}_{kind}"] for e in range(E)]) for kind in ("gate", "up", "down"))
        want = plain_experts(x, sel_e, sel_w, wg, wu, wd, base, on_output)
        err = float((out.double().cpu() - want).abs().max() / (want - base.double()).abs().max())
        assert err < 2.0 ** -8 + 2.0 ** -9, err
    assert ("experts_sums", torch.float32) in ws._buffers or not tiles
