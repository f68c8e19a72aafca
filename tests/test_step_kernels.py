"""Kernels whose form goes by the sizes and the alignment they are given: each against its formula in float64, at sizes on
both sides of every line, the vector forms also against the general ones (rows that start off a 16-byte boundary)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, PAGE = "cuda", 64


@pytest.fixture(scope="module")
def ops():
    from janus_b200.kernels import ops as o
    return o


def rnd(*shape, seed=0, s=1.0, mean=0.0):
    g = torch.Generator().manual_seed(1000 * seed + sum(shape))
    return (torch.randn(*shape, generator=g) * s + mean).to(DEV)


def worst(got, want):
    want = want.double()
    return float(((got.double() - want).abs() / (want.abs() + want.abs().mean() + 1e-30)).max())


# half a unit of bfloat16 (2^-9 of a value) and a hundred float32 roundings behind it
TOL = {torch.bfloat16: 2.0 ** -8, torch.float32: 100 * 2.0 ** -24}


def ints(*v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def pages_of(T, rows, width, dtype):
    """(cache of zeros, the cache row of each of T tokens, out of order)"""
    n = (T + PAGE - 1) // PAGE + 1
    order = torch.randperm(n * PAGE, generator=torch.Generator().manual_seed(T))[:T]
    return torch.zeros(n, rows, PAGE, width, dtype=dtype, device=DEV), order.int().to(DEV)


def table_of(positions, half):
    a = torch.arange(positions, dtype=torch.float64)[:, None] * torch.tensor([0.9 ** i for i in range(half)], dtype=torch.float64)
    return torch.stack([torch.cos(a), torch.sin(a)], -1).float().to(DEV)


def turned(x, pos, table, rot):
    if not rot:
        return x
    half = rot // 2
    c, s = table[pos.long(), :, 0].double()[:, None], table[pos.long(), :, 1].double()[:, None]
    u, v = x[..., :half], x[..., half:rot]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., rot:]], -1)


def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def picked(cache, dest):
    return cache[dest.long() // PAGE, :, dest.long() % PAGE]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H, G, d, rot", [(4, 2, 16, 8), (32, 8, 128, 64), (3, 1, 20, 0), (16, 4, 128, 128), (5, 5, 132, 8),
                                          (8, 2, 36, 12), (40, 8, 256, 128)])
@pytest.mark.parametrize("off", [0, 1])
def test_qk_norm_rope_cache(ops, H, G, d, rot, dtype, off):
    T, eps = 5, 1e-5
    wide = rnd(T, (H + G) * d + 4 + off)                     # off = 1: rows that are no whole vectors take the general kernel
    bq, bk, wq, wk = rnd(H * d, seed=1), rnd(G * d, seed=2), rnd(H * d, seed=3), rnd(G * d, seed=4)
    pos, table = ints(0, 7, 3, 90, 41), table_of(100, max(rot // 2, 1)) if rot else None
    k_cache, dest = pages_of(T, G, d, dtype)
    v_cache, q = torch.zeros_like(k_cache), torch.empty(T, H * d, dtype=dtype, device=DEV)
    ops.qk_norm_rope_cache(wide, bq, bk, wq, wk, eps, table, rot, pos, q, dest, k_cache, v_cache, H, G, d, PAGE)
    x = wide.double()
    qd, kd = x[:, :H * d] + bq.double(), x[:, H * d:(H + G) * d] + bk.double()
    want_q = turned((unit(qd, eps) * wq.double()).view(T, H, d), pos, table, rot)
    want_k = turned((unit(kd, eps) * wk.double()).view(T, G, d), pos, table, rot)
    assert worst(q.view(T, H, d), want_q) <= TOL[dtype]
    assert worst(picked(k_cache, dest), want_k) <= TOL[dtype]
    assert worst(picked(v_cache, dest), kd.view(T, G, d)) <= TOL[dtype]
    assert int((k_cache != 0).any(-1).sum()) == T * G


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T", [3, 300])
@pytest.mark.parametrize("H, G, d, e, dp, rot", [(16, 4, 128, 128, 128, 64), (4, 2, 20, 12, 24, 16), (3, 3, 128, 132, 128, 128),
                                                 (33, 1, 64, 64, 64, 0), (4, 1, 128, 64, 136, 8), (2, 2, 132, 64, 136, 8),
                                                 (4, 2, 12, 12, 16, 12)])
@pytest.mark.parametrize("form", ["weights", "unit", "mixed"])
def test_head_norm_rope_cache(ops, T, H, G, d, e, dp, rot, form, dtype):
    eps, ep = 1e-5, (e + 7) // 8 * 8
    proj = rnd(T, (H + G) * d + G * e + 4)
    pos = torch.randint(0, 500, (T,), generator=torch.Generator().manual_seed(T), dtype=torch.int32).to(DEV)
    table = table_of(500, max(rot // 2, 1)) if rot else None
    wq, wk = (rnd(d, seed=1), rnd(d, seed=2)) if form != "unit" else (None, None)
    first = rnd(T, G * e, seed=3) if form == "mixed" else None
    k_cache, dest = pages_of(T, G, dp, dtype)
    v_cache, q = torch.zeros(k_cache.shape[0], G, PAGE, ep, dtype=dtype, device=DEV), torch.full((T, H * dp), 9.0, dtype=dtype, device=DEV)
    every = 0 if form == "mixed" else 128
    ops.head_norm_rope_cache(proj, wq, wk, eps, table, rot, pos, q, dest, k_cache, v_cache, H, G, d, e, dp, PAGE,
                             unit_norm=form == "unit", temp_coef=0.1, temp_every=every, stored_vdim=ep, first=first, mix=0.3)
    x = proj.double()
    qd, kd = unit(x[:, :H * d].view(T, H, d), eps), unit(x[:, H * d:(H + G) * d].view(T, G, d), eps)
    if wq is not None:
        qd, kd = qd * wq.double(), kd * wk.double()
    vd = x[:, (H + G) * d:(H + G) * d + G * e].view(T, G, e)
    if first is not None:
        vd = 0.7 * vd + 0.3 * first.double().view(T, G, e)
    qd, kd = turned(qd, pos, table, rot), turned(kd, pos, table, rot)
    if every:
        qd = qd * (1.0 + 0.1 * torch.log(((pos.double() + 1) / every).floor() + 1.0))[:, None, None]
    got = q.view(T, H, dp)
    assert worst(got[..., :d], qd) <= TOL[dtype] and not bool(got[..., d:].any())
    assert worst(picked(k_cache, dest)[..., :d], kd) <= TOL[dtype]
    assert worst(picked(v_cache, dest)[..., :e], vd) <= TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T, Q, r, rp", [(1, 8192, 256, 256), (5, 4096, 20, 24), (3, 4100, 1024, 1024), (2, 64, 1028, 1028),
                                         (2, 61, 16, 16)])
def test_latent_prep(ops, T, Q, r, rp, dtype):
    proj, w, eps = rnd(T, Q + r), rnd(r, seed=1), 1e-5
    cache, dest = pages_of(T, 1, rp, dtype)
    q = torch.empty(T, Q, dtype=dtype, device=DEV)
    ops.latent_prep(proj, Q, r, w, eps, q, dest, cache, stored_rank=rp)
    assert torch.equal(q, proj[:, :Q].to(dtype))
    assert worst(picked(cache, dest)[:, 0, :r], unit(proj[:, Q:].double(), eps) * w.double()) <= TOL[dtype]


@pytest.mark.parametrize("T", [1, 148, 149])
@pytest.mark.parametrize("N, parts", [(1020, 1), (1024, 1), (2048, 1), (2052, 1), (4096, 2), (4100, 1), (8192, 1), (8196, 1), (16384, 4)])
def test_gated_group_rmsnorm(ops, T, N, parts):
    y, wide, w, eps = rnd(T, N), rnd(T, N + 4, seed=1), rnd(N, seed=2), 1e-5
    out = torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    ops.gated_group_rmsnorm(y, wide[:, :N], w, eps, parts, out)
    z = wide[:, :N].double()
    v = (y.double() * z * torch.sigmoid(z)).view(T, parts, -1)
    assert worst(out, unit(v, eps).view(T, N) * w.double()) <= TOL[torch.bfloat16]


@pytest.mark.parametrize("n_seqs, H, G, N, P", [(1, 2, 1, 16, 64), (3, 4, 2, 128, 64), (2, 2, 1, 100, 68), (2, 3, 3, 256, 12),
                                                (2, 2, 1, 64, 10)])
def test_mamba2_single_tokens(ops, n_seqs, H, G, N, P):
    """One token of every sequence, slots out of order: the single-token kernel (P a multiple of 4) and the walk."""
    ld = H * P + 2 * G * N
    xbc, dt, bias, a_log, skip = rnd(n_seqs, ld), rnd(n_seqs, H, seed=1), rnd(H, seed=2), rnd(H, seed=3, s=0.5), rnd(H, seed=4)
    before = rnd(n_seqs + 2, H * N * P + 8, seed=5)
    slots, q_start = torch.arange(n_seqs - 1, -1, -1, dtype=torch.int32, device=DEV), torch.arange(n_seqs + 1, dtype=torch.int32, device=DEV)
    out, state = torch.empty(n_seqs, H * P, device=DEV), before.clone()
    ops.mamba2_scan(xbc, H * P, H * P + G * N, dt, bias, a_log, skip, out, state, 4, q_start, slots, n_seqs, H, G, N, P,
                    single_tokens=True)
    walked, state2 = torch.empty_like(out), before.clone()
    ops.mamba2_scan(xbc, H * P, H * P + G * N, dt, bias, a_log, skip, walked, state2, 4, q_start, slots, n_seqs, H, G, N, P)
    x = xbc.double()
    v, b, c = x[:, :H * P].view(-1, H, P), x[:, H * P:H * P + G * N].view(-1, G, N), x[:, H * P + G * N:].view(-1, G, N)
    b, c = b.repeat_interleave(H // G, 1), c.repeat_interleave(H // G, 1)
    z = dt.double() + bias.double()
    step = torch.logaddexp(z, torch.zeros_like(z))
    old = before[slots.long(), 4:4 + H * N * P].double().view(n_seqs, H, N, P)
    new = torch.exp(-torch.exp(a_log.double()) * step)[..., None, None] * old + (step[..., None] * b)[..., None] * v[:, :, None]
    y = torch.einsum("shnp,shn->shp", new, c) + skip.double()[:, None] * v
    # sums of N products of numbers of size one, decays from exponentials: a few hundred roundings of 2^-24
    for got, st in ((out, state), (walked, state2)):
        assert worst(got.view(n_seqs, H, P), y) <= 2e-5
        assert worst(st[slots.long(), 4:4 + H * N * P].view(n_seqs, H, N, P), new) <= 2e-5
        keep = torch.ones_like(before, dtype=torch.bool)
        keep[slots.long(), 4:4 + H * N * P] = False
        assert torch.equal(st[keep], before[keep])


@pytest.mark.parametrize("H, G, d, e", [(2, 1, 128, 128), (4, 2, 64, 24), (2, 2, 20, 17), (3, 3, 4, 130)])
@pytest.mark.parametrize("lens", [[64], [65, 1, 31, 32, 33], [200, 3]])
@pytest.mark.parametrize("slab", [0, 2])
def test_delta_rule_chunks(ops, H, G, d, e, lens, slab):
    """Prompts by chunks of 32 against the recurrence in float64 and against the walk token by token, unequal lengths, slots
    out of order, from a state that is not zero, with scratch for everything or for two chunks a sequence at a time."""
    T, n = sum(lens), len(lens)
    cols = 2 * G * d + H * e
    ldc = (cols + 3) // 4 * 4
    conv, raw = rnd(T, ldc), rnd(T, 2 * H + 3, seed=1)
    a_log, bias = rnd(H, seed=2, mean=-1.0), rnd(H, seed=3)
    before = rnd(n + 1, H * d * e + 4, seed=4, s=0.3)
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slots = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    floats = (slab or (max(lens) + 31) // 32) * n * H * ops._DELTA_CHUNK_FLOATS
    asked = ops.delta_rule_scratch(n, H, max(lens), ldc, 0, G * d, d)
    assert asked == (0 if d <= 64 or max(lens) < 192 else n * H * 7 * ops._DELTA_CHUNK_FLOATS)
    results = []
    for scratch in (torch.full((floats,), float("nan"), device=DEV), None):
        out, state = torch.full((T, H * e), float("nan"), device=DEV), before.clone()
        ops.delta_rule(conv, 0, G * d, 2 * G * d, raw, 0, H, a_log, bias, 1e-6, out, state, 4, q_start, slots, n, H, G, d, e,
                       scratch, max(lens))
        results.append((out, state))
    x = conv.double()
    q, k, v = x[:, :G * d].view(T, G, d), x[:, G * d:2 * G * d].view(T, G, d), x[:, 2 * G * d:cols].reshape(T, H, e)
    norm = lambda t: (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)      # noqa: E731
    q, k = norm(q) * d ** -0.5, norm(k)
    beta = torch.sigmoid(raw[:, :H].double())
    z = raw[:, H:2 * H].double() + bias.double()
    decay = torch.exp(-torch.exp(a_log.double()) * torch.logaddexp(z, torch.zeros_like(z)))
    want, after = torch.zeros(T, H, e, dtype=torch.float64, device=DEV), before.double().clone()
    at = 0
    for s, length in enumerate(lens):
        S = before[slots[s].long(), 4:].double().view(H, d, e)
        for t in range(at, at + length):
            S = decay[t][:, None, None] * S
            w = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
            S = S + k[t][:, :, None] * w[:, None, :]
            want[t] = torch.einsum("hde,hd->he", S, q[t])
        after[slots[s].long(), 4:] = S.reshape(-1)
        at += length
    # sums of up to 128 products and a chain of 32 writes a chunk, decays that forget what lies far back: a few hundred
    # roundings of 2^-24 against the mean size of a result; the walk's own error stands beside it
    err = [max(worst(o.view(T, H, e), want), worst(s, after)) for o, s in results]
    assert err[0] <= 4e-5 and err[0] <= 4 * err[1] + 4e-6, err


@pytest.mark.parametrize("H, G, d, e", [(4, 1, 64, 128), (4, 2, 16, 64), (2, 2, 72, 72), (3, 1, 128, 8)])
@pytest.mark.parametrize("window, kept", [(0, 0), (40, 0), (512, 4), (512, 70), (1, 33)])
@pytest.mark.parametrize("copies", [1, 60])
def test_diff_attention_single_tokens(ops, H, G, d, e, window, kept, copies):
    """One query of every sequence over bfloat16 pages, lengths at the edges of chunks (32) and pages (64), windows that
    start inside a chunk, kept keys in their own chunk or in the window's, few pairs and many (fewer warps a pair)."""
    lens = [1, 32, 33, 64, 97, 600, 745] * copies
    B, n_pages = len(lens), sum((n + PAGE - 1) // PAGE for n in lens)
    g = torch.Generator().manual_seed(d + e)
    kc = torch.randn(n_pages, 2 * G, PAGE, d, generator=g).to(torch.bfloat16).to(DEV)
    vc = torch.randn(n_pages, G, PAGE, e, generator=g).to(torch.bfloat16).to(DEV)
    order, at = torch.randperm(n_pages, generator=g), 0
    table = torch.full((B, 12), -1, dtype=torch.int32)
    for b, n in enumerate(lens):
        need = (n + PAGE - 1) // PAGE
        table[b, :need] = order[at:at + need].int()
        at += need
    table = table.to(DEV)
    q = rnd(B, H * 2 * d)
    pos, seq = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), torch.arange(B, dtype=torch.int32, device=DEV)
    out = torch.empty(B, H * e, dtype=torch.bfloat16, device=DEV)
    lam, eps, scale = 0.4, 1e-5, d ** -0.5
    ops.diff_attention(q, kc, vc, out, table, seq, pos, H, G, d, e, PAGE, window, kept, scale, lam, eps, 0.5)
    for b in range(7):
        n = lens[b]
        pages = table[b, :(n + PAGE - 1) // PAGE].long()
        k = kc[pages].double().permute(1, 0, 2, 3).reshape(G, 2, -1, d)[:, :, :n]
        v = vc[pages].double().permute(1, 0, 2, 3).reshape(G, -1, e)[:, :n]
        j = torch.arange(n, device=DEV)
        seen = (n - 1 - j < window) | (j < kept) if window else torch.ones(n, dtype=torch.bool, device=DEV)
        qq = q[b].double().view(H, 2, d)
        s = torch.einsum("hmd,hmnd->hmn", qq, k.repeat_interleave(H // G, 0)) * scale
        p = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
        maps = torch.einsum("hmn,hne->hme", p, v.repeat_interleave(H // G, 0))
        want = unit(maps[:, 0] - lam * maps[:, 1], eps) * 0.5
        # scores of size one from float32 sums of up to 128 products, then bfloat16; a difference that nearly cancels is
        # divided by its own size, hence the room of a factor of four
        assert worst(out[b].view(H, e), want) <= 4 * TOL[torch.bfloat16]
    for b in range(7, B):
        if b % 7 == 3:
            assert bool(torch.isfinite(out[b].float()).all())


def conv_reference(x, w, lens, states):
    """x [T, C] float64 of sequences of the given lengths, w [C, taps], states [n, taps - 1, C]: the causal convolution."""
    taps, out, at = w.shape[1], [], 0
    for n, st in zip(lens, states):
        full = torch.cat([st, x[at:at + n]])
        out.append(sum(full[j:j + n] * w[:, j] for j in range(taps)))
        at += n
    return torch.cat(out)


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("C", [8, 516])
@pytest.mark.parametrize("lens", [[64], [1, 15, 2, 47, 16], [130, 1, 1, 1, 17]])
def test_causal_conv_silu_prompts(ops, taps, C, lens):
    """Walks of sixteen tokens with eight (four taps) or four inputs in flight; sequences that begin and end inside a walk."""
    T, n = sum(lens), len(lens)
    x, w, bias = rnd(T, C + 4), rnd(C, taps, seed=1), rnd(C, seed=2)
    state = rnd(n + 1, (taps - 1) * C + 4, seed=3)
    slots = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(lens)).int().to(DEV)
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    before, out = state.double().clone(), torch.empty(T, C, device=DEV)
    ops.causal_conv_silu(x, 4, C, w, bias, taps, state, 4, seq, q_start, slots, out, n)
    states = [before[s, 4:].view(taps - 1, C) for s in slots.tolist()]
    y = conv_reference(x[:, 4:].double(), w.double(), lens, states) + bias.double()
    assert worst(out, y * torch.sigmoid(y)) <= TOL[torch.float32]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("H, G, d, e, rot", [(4, 2, 64, 128, 32), (2, 1, 16, 12, 16), (3, 3, 20, 8, 0), (2, 2, 12, 20, 8)])
@pytest.mark.parametrize("lens", [[63], [1, 15, 2, 47, 16], [130, 1, 1, 1, 17]])
def test_conv_rope_cache_prompts(ops, H, G, d, e, rot, taps, lens, dtype):
    """Prompts of 64 tokens and more walk with their inputs in registers where there are two to four taps, others take a
    token a thread; sequences that begin and end inside a walk, states that are not zero."""
    T, n, C = sum(lens), len(lens), H * 2 * d + G * 2 * d + G * e
    proj, w = rnd(T, C), rnd(C, max(taps, 1), seed=1) if taps else None
    state = rnd(n + 1, max(taps - 1, 1), C, seed=3)
    slots = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(lens)).int().to(DEV)
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(k) + 3 for k in lens]).int().to(DEV)
    table = table_of(200, rot // 2) if rot else None
    k_cache, dest = pages_of(T, 2 * G, d, dtype)
    v_cache, q = torch.zeros(k_cache.shape[0], G, PAGE, e, dtype=dtype, device=DEV), torch.empty(T, H * 2 * d, device=DEV)
    ops.conv_rope_cache(proj, w, taps if taps else 1, state if taps else None, seq, q_start, slots, pos, table, rot, q, dest, k_cache,
                        v_cache, H, G, d, e, PAGE)
    x = proj.double()
    if taps:
        x = conv_reference(x, w.double(), lens, [state[s].double() for s in slots.tolist()])
    want_q = turned(x[:, :H * 2 * d].view(T, 2 * H, d), pos, table, rot)
    want_k = turned(x[:, H * 2 * d:(H + G) * 2 * d].view(T, 2 * G, d), pos, table, rot)
    assert worst(q.view(T, 2 * H, d), want_q) <= TOL[torch.float32]
    assert worst(picked(k_cache, dest), want_k) <= TOL[dtype]
    assert worst(picked(v_cache, dest), x[:, (H + G) * 2 * d:].view(T, G, e)) <= TOL[dtype]


@pytest.mark.parametrize("T", [1, 296, 297])
@pytest.mark.parametrize("N", [508, 512, 2048, 2052, 4096, 4100])
def test_gated_rmsnorm(ops, T, N):
    o, wide, w, eps = rnd(T, N), rnd(T, N + 4, seed=1), rnd(N, seed=2).to(torch.bfloat16), 1e-5
    out = torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    ops.gated_rmsnorm(o, w, wide[:, :N], eps, out)
    assert worst(out, unit(o.double(), eps) * w.double() * torch.sigmoid(wide[:, :N].double())) <= TOL[torch.bfloat16]


@pytest.mark.parametrize("rank", [1, 15, 16, 17, 64, 66])
@pytest.mark.parametrize("T, C", [(1, 7), (8, 2048), (17, 515)])
def test_gla_decay(ops, T, C, rank):
    proj, a2, bias = rnd(T, rank + 5), rnd(C, rank, seed=1), rnd(C, seed=2)
    alpha = torch.empty(T, C, device=DEV)
    ops.gla_decay(proj, 5, rank, a2.t().contiguous(), bias, 16.0, alpha)
    z = proj[:, 5:].double() @ a2.double().T + bias.double()
    # the argument's error (rank roundings of a sum of the size sqrt(rank)) reaches a decay through a sixteenth of itself
    assert worst(alpha, torch.sigmoid(z) ** (1 / 16.0)) <= TOL[torch.float32]


@pytest.mark.parametrize("n_seqs, H, d, e", [(1, 2, 16, 64), (3, 4, 128, 128), (2, 2, 100, 68), (2, 3, 256, 12), (2, 2, 64, 10)])
@pytest.mark.parametrize("kind", ["channels", "normalizer"])
def test_state_steps(ops, n_seqs, H, d, e, kind):
    """One token of every sequence, slots out of order: the single-token kernels (values a multiple of 4) and the walks."""
    ld = H * (2 * d + e)
    proj = rnd(n_seqs, ld)
    slots, q_start = torch.arange(n_seqs - 1, -1, -1, dtype=torch.int32, device=DEV), torch.arange(n_seqs + 1, dtype=torch.int32, device=DEV)
    per = d * (e + 1) if kind == "normalizer" else d * e
    before = rnd(n_seqs + 1, H * per, seed=5)
    q, k, v = proj[:, :H * d].double().view(-1, H, d), proj[:, H * d:2 * H * d].double().view(-1, H, d), proj[:, 2 * H * d:].double().view(-1, H, e)
    old = before[slots.long()].double().view(n_seqs, H, per)
    S, scale, den, gates = old[..., :d * e].view(n_seqs, H, d, e), d ** -0.5, None, None
    if kind == "channels":
        gates = torch.rand(n_seqs, H * d, generator=torch.Generator().manual_seed(2)).to(DEV)
        a = gates.double().view(n_seqs, H, d)
    else:
        gates = torch.rand(n_seqs, H, 4, generator=torch.Generator().manual_seed(2)).to(DEV)
        a, v = gates[..., 0:1].double(), v * gates[..., 1:2].double()
        n = a * old[..., d * e:] + gates[..., 1:2].double() * k
        den = torch.maximum((n * q).sum(-1).abs() * scale, gates[..., 2].double()) + 1e-6
    new = a[..., None] * S + k[..., None] * v[:, :, None]
    y = torch.einsum("shde,shd->she", new, q) * scale
    for single in (True, False):
        out, state = torch.empty(n_seqs, H * e, device=DEV), before.clone()
        got_den = torch.empty(n_seqs, H, device=DEV) if den is not None else None
        ops.gated_linear_scan(proj, 0, H * d, 2 * H * d, scale, gates, out, state, q_start, slots, n_seqs, H, d, e,
                              divisors=got_den, single_tokens=single)
        # sums of d products of numbers of size one: a few hundred roundings of 2^-24
        got = state[slots.long()].view(n_seqs, H, per)
        assert worst(out.view(n_seqs, H, e), y) <= 2e-5
        assert worst(got[..., :d * e].reshape(n_seqs, H, d, e), new) <= 2e-5
        if den is not None:
            assert worst(got[..., d * e:], n) <= 2e-5 and worst(got_den, den) <= 2e-5
        assert torch.equal(state[n_seqs], before[n_seqs])


class Scratch:
    def __init__(self):
        self.asked = []

    def get(self, name, shape, dtype):
        self.asked.append(name)
        return torch.full(shape, float("nan"), dtype=dtype, device=DEV)


@pytest.mark.parametrize("H, G, d, e", [(2, 2, 128, 128), (4, 4, 64, 24), (3, 3, 20, 17), (2, 2, 4, 33), (6, 6, 128, 66), (2, 2, 68, 64), (2, 2, 64, 130), (76, 76, 72, 66)])
@pytest.mark.parametrize("lens", [[64], [65, 1, 31, 32, 33], [300, 3]])
@pytest.mark.parametrize("kind", ["mamba", "lightning", "memory"])
@pytest.mark.parametrize("slab", [0, 2])
def test_state_chunks(ops, monkeypatch, H, G, d, e, lens, kind, slab):
    """Prompts by chunks of 32 tokens against the recurrences in float64 and against the walk token by token: unequal lengths,
    slots out of order, states that are not zero, decays of zero and of one, scratch for everything or two chunks at a time."""
    G = {"mamba": max(1, H // 2) if H % 2 == 0 else 1}.get(kind, H)
    T, n = sum(lens), len(lens)
    if slab:
        monkeypatch.setattr(ops, "STATE_SCRATCH_BYTES", slab * n * H * 4 * ops._STATE_KINDS[kind][1])
    monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: True)
    per = d * (e + 1) if kind == "memory" else d * e
    before = rnd(n + 1, H * per + (4 if kind == "mamba" else 0), seed=4, s=0.3)
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slots = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    vw = (H * e + 3) // 4 * 4
    proj = rnd(T, vw + 2 * G * d)
    v, k, q = proj[:, :H * e].double().view(T, H, e), proj[:, vw:vw + G * d].double(), proj[:, vw + G * d:].double()
    k, q = (t.view(T, G, d).repeat_interleave(H // G, 1) for t in (k, q))
    silu = lambda z: z * torch.sigmoid(z)                                                                      # noqa: E731
    scale, skip = 1.0, torch.zeros(H, device=DEV)
    g = torch.Generator().manual_seed(7)
    if kind == "mamba":
        raw, bias, a_log, skip = rnd(T, H, seed=5), rnd(H, seed=6), rnd(H, seed=7, s=0.5), rnd(H, seed=8)
        z = raw.double() + bias.double()
        take = torch.logaddexp(z, torch.zeros_like(z))
        keep = torch.exp(-torch.exp(a_log.double()) * take)
    elif kind == "lightning":
        decay = torch.tensor([[0.97, 1.0, 0.3, 0.999, 0.5, 0.0][h % 6] for h in range(H)], device=DEV)
        keep, take = decay.double().expand(T, H), torch.ones(T, H, dtype=torch.float64, device=DEV)
        q, k, v = silu(q), silu(k), silu(v)
    else:
        gates = torch.rand(T, H, 4, generator=g)
        gates[:, :, 0] = gates[:, :, 0] ** 0.2
        gates[3::17, :, 0] = 0.0
        gates, scale = gates.to(DEV), d ** -0.5
        keep, take = gates[..., 0].double(), gates[..., 1].double()
    results = []
    for workspace in (Scratch(), None):
        out, state = torch.full((T, H * e), float("nan"), device=DEV), before.clone()
        den = torch.full((T, H), float("nan"), device=DEV) if kind == "memory" else None
        if kind == "mamba":
            ops.mamba2_scan(proj, vw, vw + G * d, raw, bias, a_log, skip, out, state, 4, q_start, slots, n, H, G, d, e, max(lens), workspace)
        elif kind == "lightning":
            ops.lightning_scan(proj, vw + G * d, vw, 0, out, state.view(-1, H, d, e), q_start, slots, decay, n, H, d, e, max(lens), workspace)
        else:
            ops.gated_linear_scan(proj, vw + G * d, vw, 0, scale, gates, out, state, q_start, slots, n, H, d, e, max(lens), workspace,
                                  divisors=den)
        assert workspace is None or workspace.asked == ["state_chunks"]
        results.append((out, state, den))
    off = 4 if kind == "mamba" else 0
    want, after, want_den = torch.zeros(T, H, e, dtype=torch.float64, device=DEV), before.double().clone(), torch.zeros(T, H, dtype=torch.float64, device=DEV)
    at = 0
    for s, length in enumerate(lens):
        st = before[slots[s].long(), off:].double().view(H, per)
        S, norm = st[:, :d * e].view(H, d, e), st[:, d * e:]
        for t in range(at, at + length):
            S = keep[t][:, None, None] * S + (take[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hde,hd->he", S, q[t]) * scale + skip.double()[:, None] * v[t]
            if kind == "memory":
                norm = keep[t][:, None] * norm + take[t][:, None] * k[t]
                want_den[t] = torch.maximum((norm * q[t]).sum(-1).abs() * scale, gates[t, :, 2].double()) + 1e-6
        after[slots[s].long(), off:] = torch.cat([S.reshape(H, -1), norm], 1).reshape(-1)
        at += length
    # sums of up to 128 products, states that grow where nothing decays: some hundred roundings of 2^-24 against the mean size
    # of a result; the walk's own error stands beside it
    err = [max(worst(o.view(T, H, e), want), worst(st, after), worst(dn, want_den) if dn is not None else 0.0) for o, st, dn in results]
    assert err[0] <= 6e-5 and err[0] <= 4 * err[1] + 4e-6, err


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H", [6, 8, 2044, 2048])
@pytest.mark.parametrize("T", [1, 297])
def test_embed_streams(ops, T, H, dtype):
    """Every stream starts as the token's row: a copy, number for number."""
    table, ids = rnd(50, H).to(dtype), torch.randint(0, 50, (T,), dtype=torch.int32, device=DEV)
    out = torch.full((T, 3 * H), float("nan"), device=DEV)
    ops.embed_streams(table, ids, out, 3)
    assert torch.equal(out.view(T, 3, H), table[ids.long()].float()[:, None].expand(T, 3, H))


@pytest.mark.parametrize("T, W, E", [(16, 1184, 8), (16, 1216, 8), (1, 2048, 4), (3, 4736, 4)])
def test_expert_down_blocks(ops, T, W, E):
    """The second product of few pairs' experts on both sides of the line between few blocks and many."""
    F, top = 96, 2
    h = rnd(T, W, s=W ** -0.5).bfloat16()
    wg, wu, wd = (rnd(E, *s, seed=i + 1).bfloat16() for i, s in enumerate(((F, W), (F, W), (W, F))))
    sel = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:top] for t in range(T)]).int().to(DEV)
    weight = rnd(T, top, seed=9).abs() + 0.2
    out, act = torch.zeros(T, W, device=DEV), torch.empty(T * top, F, dtype=torch.bfloat16, device=DEV)
    ops.experts_few_tokens_tc(h, sel, weight, wg, wu, wd, act, out, weight_on_output=True)
    want, bound = (torch.zeros(T, W, dtype=torch.float64, device=DEV) for _ in range(2))
    for t in range(T):
        for j in range(top):
            e, w = int(sel[t, j]), weight[t, j].double()
            gate, up = wg[e].double() @ h[t].double(), wu[e].double() @ h[t].double()
            between = gate * torch.sigmoid(gate) * up
            want[t] += wd[e].double() @ between * w
            bound[t] += wd[e].double().abs() @ between.abs() * w
    # what stands between the products is rounded to bfloat16: half of 2^-8 of each number, and the float32 sums
    assert bool(((out.double() - want).abs() <= (2.0 ** -9 + 2.0 ** -12) * bound).all())


def lightning_reference(q, k, v, decay, before, lens, slots):
    """(outputs, states) of S <- decay S + k v^T, y = S^T q in float64; q, k, v [T, H, .] activated"""
    out, after, at = torch.zeros(*v.shape, dtype=torch.float64, device=DEV), before.double().clone(), 0
    for s, length in enumerate(lens):
        S = before[slots[s].long()].double()
        for t in range(at, at + length):
            S = decay.double()[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hde,hd->he", S, q[t])
        after[slots[s].long()] = S
        at += length
    return out, after


@pytest.mark.parametrize("length", [64, 300])
@pytest.mark.parametrize("d", [64, 128])
def test_lightning_decays_of_any_sign(ops, monkeypatch, length, d):
    """Decays below zero, above one and zero with either sign: chunks take them as the walk does."""
    decay = torch.tensor([-0.5, 1.05, 0.9, -1.02, -0.0, -0.999], device=DEV)
    H, e, lens = decay.numel(), 64, [length, 40]
    T = sum(lens)
    proj, before = rnd(T, H * (2 * d + e)), rnd(3, H, d, e, seed=4, s=0.3)
    q_start, slots = ints(0, length, T), ints(2, 0)
    q, k, v = (torch.nn.functional.silu(t.double()).view(T, H, -1) for t in proj.split([H * d, H * d, H * e], 1))
    want, after = lightning_reference(q, k, v, decay, before, lens, slots)
    for pays, asked in ((True, ["state_chunks"]), (False, [] if length <= 256 else ["lightning_segments"])):
        monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: pays)
        out, state, workspace = torch.full((T, H * e), float("nan"), device=DEV), before.clone(), Scratch()
        ops.lightning_scan(proj, 0, H * d, 2 * H * d, out, state, q_start, slots, decay, 2, H, d, e, length, workspace)
        assert workspace.asked == asked
        for h in range(H):                                   # some hundred roundings of 2^-24 against the head's mean size
            assert worst(out.view(T, H, e)[:, h], want[:, h]) <= 4e-5, (pays, h)
            assert worst(state[:, h], after[:, h]) <= 4e-5, (pays, h)


@pytest.mark.parametrize("kind", ["mamba", "lightning", "memory", "delta"])
def test_an_infinite_value_stays_behind_its_token(ops, monkeypatch, kind):
    """An infinity among a token's values reaches its own column from that token on, whichever place of a chunk the token has:
    everything else keeps every bit, by chunks as by the walk."""
    H, d, e, lens, places = 2, 128, 64, [200, 70], [(64, 3), (66, 7), (77, 40), (94, 11), (95, 60), (201, 5)]
    T, per = sum(lens), 128 * 64 + (128 if kind == "memory" else 0)
    q_start, slots = ints(0, 200, T), ints(1, 0)
    before, raw, bias, rate = rnd(2, H * per, seed=1, s=0.3), rnd(T, 2 * H, seed=2), rnd(H, seed=3), rnd(H, seed=4, mean=-1.0)
    decay, gates = torch.tensor([0.9, 0.99], device=DEV), torch.rand(T, H, 4, generator=torch.Generator().manual_seed(5)).to(DEV)
    monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: True)
    # the chunks by the size of a block (two or four parts share its sums), then the walk
    for chunks, copies in ((True, 1), (True, 80), (False, 1)):
        many, n = torch.arange(copies).repeat_interleave(2).mul(270).to(DEV), 2 * copies
        starts = torch.cat([q_start[:2].repeat(copies) + many, many.new_full((1,), 270 * copies)]).int()
        where = torch.arange(n, device=DEV).int()
        results = []
        for inf in (True, False):
            one = rnd(T, H * (2 * d + e))
            for t, c in places if inf else ():
                one[t, 2 * H * d + c] = float("inf")
            proj, out = one.repeat(copies, 1), torch.zeros(copies * T, H * e, device=DEV)
            state, workspace = before[slots.long()].repeat(copies, 1), Scratch() if chunks else None
            if kind == "mamba":
                ops.mamba2_scan(torch.cat([proj[:, 2 * H * d:], proj[:, :2 * H * d]], 1), H * e, H * (e + d), raw.repeat(copies, 1)[:, :H], bias, rate,
                                bias, out, state, 0, starts, where, n, H, H, d, e, 200, workspace)
            elif kind == "lightning":
                ops.lightning_scan(proj, 0, H * d, 2 * H * d, out, state.view(n, H, d, e), starts, where, decay, n, H, d, e, 200, workspace)
            elif kind == "memory":
                ops.gated_linear_scan(proj, 0, H * d, 2 * H * d, 1.0, gates.repeat(copies, 1, 1), out, state, starts, where, n, H, d, e, 200,
                                      workspace, divisors=torch.empty(copies * T, H, device=DEV))
            else:
                floats = H * n * 7 * ops._DELTA_CHUNK_FLOATS
                ops.delta_rule(proj, 0, H * d, 2 * H * d, raw.repeat(copies, 1), 0, H, rate, bias, 1e-6, out, state, 0, starts, where, n, H, H, d,
                               e, torch.full((floats,), float("nan"), device=DEV) if chunks else None, 200)
            results.append(out.view(copies, T, H, e))
        got, clean = results
        for t, c in places:
            end = 200 if t < 200 else T
            assert not bool(torch.isfinite(got[:, t:end, 0, c]).any()), (chunks, copies, t)
            got[:, t:end, 0, c] = clean[:, t:end, 0, c]
        assert torch.equal(got, clean), (chunks, copies)


@pytest.mark.parametrize("kind", ["mamba", "lightning", "memory", "delta"])
def test_a_nan_decay_shows(ops, monkeypatch, kind):
    """A decay that is not a number makes its head's outputs from that token on not a number, by chunks as by the walk; the
    tokens before it, the other head and the other sequence keep every bit."""
    H, d, e, lens, bad = 2, 128, 64, [200, 70], 77
    T, per = sum(lens), 128 * 64 + (128 if kind == "memory" else 0)
    q_start, slots = ints(0, 200, T), ints(1, 0)
    proj, before = rnd(T, H * (2 * d + e)), rnd(2, H * per, seed=1, s=0.3)
    raw, bias, rate = rnd(T, 2 * H, seed=2), rnd(H, seed=3), rnd(H, seed=4, mean=-1.0)
    gates = torch.rand(T, H, 4, generator=torch.Generator().manual_seed(5)).to(DEV)
    monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: True)
    results = {}
    for chunks in (True, False):
        for nan in (True, False):
            out, state, workspace = torch.zeros(T, H * e, device=DEV), before.clone(), Scratch() if chunks else None
            x, g, r = raw.clone(), gates.clone(), rate.clone()
            first = 0 if kind == "lightning" else bad             # a lightning layer's decays are not a token's
            if nan:
                x[bad, 0] = x[bad, H] = g[bad, 0, 0] = float("nan")
                r[0] = float("nan") if kind == "lightning" else r[0]
            if kind == "mamba":
                ops.mamba2_scan(proj, H * e, H * (e + d), x[:, :H], bias, r, bias, out, state, 0, q_start, slots, 2, H, H, d, e, 200, workspace)
            elif kind == "lightning":
                ops.lightning_scan(proj, 0, H * d, 2 * H * d, out, state.view(2, H, d, e), q_start, slots, r, 2, H, d, e, 200, workspace)
            elif kind == "memory":
                ops.gated_linear_scan(proj, 0, H * d, 2 * H * d, 1.0, g, out, state, q_start, slots, 2, H, d, e, 200, workspace,
                                      divisors=torch.empty(T, H, device=DEV))
            else:
                floats = H * 2 * 7 * ops._DELTA_CHUNK_FLOATS
                ops.delta_rule(proj, 0, H * d, 2 * H * d, x, 0, H, r, bias, 1e-6, out, state, 0, q_start, slots, 2, H, H, d, e,
                               torch.full((floats,), float("nan"), device=DEV) if chunks else None, 200)
            results[chunks, nan] = out.view(T, H, e), state.view(2, H, per)
        (out, state), (clean, clean_state) = results[chunks, True], results[chunks, False]
        sick = torch.zeros(T, H, dtype=torch.bool, device=DEV)
        sick[first:200, 0] = True
        if kind == "lightning":
            sick[:, 0] = True
        assert bool(torch.isnan(out[sick]).all()) and torch.equal(out[~sick], clean[~sick]), chunks
        assert bool(torch.isnan(state[1, 0, :d * e]).all()) and torch.equal(state[:, 1], clean_state[:, 1]), chunks


@pytest.mark.parametrize("taps", [2, 3, 4])
def test_conv_rope_cache_reaches_its_taps_only(ops, taps):
    """An infinity at a token reaches `taps` tokens of its channel, no later one, in a prompt that walks (64 tokens and more)."""
    T, H, G, d, e, bad = 80, 2, 1, 16, 16, [(20, 3), (33, 40), (47, 70)]
    C = H * 2 * d + G * 2 * d + G * e
    w, state, results = rnd(C, taps, seed=1), rnd(1, taps - 1, C, seed=2), []
    for inf in (True, False):
        proj = rnd(T, C)
        for t, c in bad if inf else ():
            proj[t, c] = float("inf")
        k_cache, dest = pages_of(T, 2 * G, d, torch.float32)
        v_cache, q = torch.zeros(k_cache.shape[0], G, PAGE, e, device=DEV), torch.empty(T, H * 2 * d, device=DEV)
        ops.conv_rope_cache(proj, w, taps, state, torch.zeros(T, dtype=torch.int32, device=DEV), ints(0, T), ints(0),
                            torch.arange(T, dtype=torch.int32, device=DEV), None, 0, q, dest, k_cache, v_cache, H, G, d, e, PAGE)
        results.append(torch.cat([q, picked(k_cache, dest).reshape(T, -1), picked(v_cache, dest).reshape(T, -1)], 1))
    got, clean = results
    for t, c in bad:
        assert not bool(torch.isfinite(got[t:t + taps, c]).any())
        got[t:t + taps, c] = clean[t:t + taps, c]
    assert torch.equal(got, clean)


def test_chunks_of_many_sequences(ops, monkeypatch):
    """A step of 300 sequences of one to 70 tokens, whose chunks lie one after another in the scratch: state space and delta
    rule against the walk (the forms' own errors against float64 are tested above)."""
    lens = [(1, 33, 2, 32, 64, 1, 70, 31)[i % 8] for i in range(300)]
    n, T, H, d, e = 300, sum(lens), 2, 68, 20
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slots = torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEV)
    proj, raw, bias, rate = rnd(T, H * (2 * d + e)), rnd(T, 2 * H, seed=1), rnd(H, seed=2), rnd(H, seed=3, mean=-1.0)
    before = rnd(n, H * d * e, seed=4, s=0.3)
    monkeypatch.setattr(ops, "state_chunks_pay", lambda *_: True)
    results = []
    for workspace in (Scratch(), None):
        out, state = torch.full((T, H * e), float("nan"), device=DEV), before.clone()
        ops.mamba2_scan(proj, H * e, H * (e + d), raw[:, :H].contiguous(), bias, rate, bias, out, state, 0, q_start, slots, n, H, H, d, e, 70, workspace)
        results.append((out, state))
    assert worst(results[0][0], results[1][0]) <= 6e-5 and worst(results[0][1], results[1][1]) <= 6e-5
    results = []
    for slots_of in (T // 32 + n, 2 * n, 0):
        out, state = torch.full((T, H * e), float("nan"), device=DEV), before.clone()
        scratch = torch.full((slots_of * H * ops._DELTA_CHUNK_FLOATS,), float("nan"), device=DEV) if slots_of else None
        ops.delta_rule(proj, 0, H * d, 2 * H * d, raw, 0, H, rate, bias, 1e-6, out, state, 0, q_start, slots, n, H, H, d, e, scratch, 70)
        results.append((out, state))
    for got in results[:2]:
        assert worst(got[0], results[2][0]) <= 4e-5 and worst(got[1], results[2][1]) <= 4e-5


@pytest.mark.parametrize("lens, chunks", [([4096] + [1] * 31, False), ([1024] * 8 + [1] * 24, True), ([200] + [1] * 63, False),
                                          ([1024, 1024], True), ([1, 1, 1500, 1], False)])
def test_mixed_steps_take_the_form_of_their_work(ops, lens, chunks):
    """What decides between walk and chunks is the work that exists: one long prompt among single tokens has the blocks of
    one sequence, and single tokens alone are no reason for chunks."""
    n, T, H, d, e = len(lens), sum(lens), 16, 128, 128
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    proj, out = rnd(T, H * (2 * d + e)), torch.empty(T, H * e, device=DEV)
    state, workspace = torch.zeros(n, H, d, e, device=DEV), Scratch()
    ops.lightning_scan(proj, 0, H * d, 2 * H * d, out, state, q_start, torch.arange(n, dtype=torch.int32, device=DEV),
                       torch.full((H,), 0.9, device=DEV), n, H, d, e, max(lens), workspace)
    assert ("state_chunks" in workspace.asked) == chunks


@pytest.mark.parametrize("W, E", [(2368, 2), (2400, 2)])
def test_expert_down_blocks_of_one_wave(ops, W, E):
    """The second product at 296 blocks, two an SM, and at 300."""
    test_expert_down_blocks(ops, 1, W, E)


@pytest.mark.parametrize("H, G, lens, slab", [(8, 2, [1600, 1500], 0), (32, 2, [2400], 0), (20, 2, [70, 33], 0), (12, 12, [700, 650, 1], 3)])
def test_delta_rule_chunks_of_many_heads(ops, H, G, lens, slab):
    """Blocks that prepare several heads of a group (two to eight, and groups of more than eight in several blocks), with
    decays that underflow to zero within a chunk and forget all before, against the walk and the walk against float64."""
    T, n, d, e = sum(lens), len(lens), 128, 40
    conv, raw = rnd(T, 2 * G * d + H * e), rnd(T, 2 * H, seed=1)
    raw[13::29, H:] = 300.0                                   # a decay of exp(-100) and less at every 29th token
    a_log, bias, before = rnd(H, seed=2, mean=-1.0), rnd(H, seed=3), rnd(n, H * d * e, seed=4, s=0.3)
    q_start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slots = torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEV)
    results = []
    for floats in ((slab or (max(lens) + 31) // 32) * n * H * ops._DELTA_CHUNK_FLOATS, 0):
        out, state = torch.full((T, H * e), float("nan"), device=DEV), before.clone()
        ops.delta_rule(conv, 0, G * d, 2 * G * d, raw, 0, H, a_log, bias, 1e-6, out, state, 0, q_start, slots, n, H, G, d, e,
                       torch.full((floats,), float("nan"), device=DEV) if floats else None, max(lens))
        results.append((out, state))
    x = conv.double()
    norm = lambda t: (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)      # noqa: E731
    q, k = norm(x[:, :G * d].view(T, G, d)) * d ** -0.5, norm(x[:, G * d:2 * G * d].view(T, G, d))
    v, beta, z = x[:, 2 * G * d:].reshape(T, H, e), torch.sigmoid(raw[:, :H].double()), raw[:, H:].double() + bias.double()
    decay = torch.exp(-torch.exp(a_log.double()) * torch.logaddexp(z, torch.zeros_like(z)))
    want, after, at = torch.zeros(T, H, e, dtype=torch.float64, device=DEV), before.double().clone(), 0
    for s, length in enumerate(lens):
        S = before[slots[s].long()].double().view(H, d, e)
        for t in range(at, at + length):
            S = decay[t][:, None, None] * S
            w = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
            S = S + k[t][:, :, None] * w[:, None, :]
            want[t] = torch.einsum("hde,hd->he", S, q[t])
        after[slots[s].long()] = S.reshape(-1)
        at += length
    # as for the sizes above: a few hundred roundings of 2^-24 against the mean size of a result
    err = [max(worst(o.view(T, H, e), want), worst(s, after)) for o, s in results]
    assert err[0] <= 4e-5 and err[0] <= 4 * err[1] + 4e-6, err


@pytest.mark.parametrize("e", [64, 128])
@pytest.mark.parametrize("window, n", [(448, 600), (512, 600), (544, 640), (576, 640), (0, 512), (0, 513), (0, 640), (0, 641)])
def test_diff_attention_rounds(ops, e, window, n):
    """One sequence whose query sees 15 to 21 chunks of 32 keys: 16 warps, or one round of 17 to 20."""
    H, G, d, kept, pages = 2, 1, 16, 4, (n + PAGE - 1) // PAGE
    g = torch.Generator().manual_seed(n + window + e)
    kc = torch.randn(pages, 2 * G, PAGE, d, generator=g).to(torch.bfloat16).to(DEV)
    vc = torch.randn(pages, G, PAGE, e, generator=g).to(torch.bfloat16).to(DEV)
    table = torch.randperm(pages, generator=g).int()[None].to(DEV)
    q, out = rnd(1, H * 2 * d), torch.empty(1, H * e, dtype=torch.bfloat16, device=DEV)
    ops.diff_attention(q, kc, vc, out, table, ints(0), ints(n - 1), H, G, d, e, PAGE, window, kept, 0.25, 0.4, 1e-5, 0.5)
    k = kc[table[0].long()].double().permute(1, 0, 2, 3).reshape(G, 2, -1, d)[:, :, :n]
    v = vc[table[0].long()].double().permute(1, 0, 2, 3).reshape(G, -1, e)[:, :n]
    j = torch.arange(n, device=DEV)
    seen = (n - 1 - j < window) | (j < kept) if window else torch.ones(n, dtype=torch.bool, device=DEV)
    s = torch.einsum("hmd,hmnd->hmn", q.double().view(H, 2, d), k.repeat_interleave(H // G, 0)) * 0.25
    maps = torch.einsum("hmn,hne->hme", torch.softmax(s.masked_fill(~seen, -math.inf), -1), v.repeat_interleave(H // G, 0))
    # bfloat16, and a difference that nearly cancels, as above
    assert worst(out.view(H, e), unit(maps[:, 0] - 0.4 * maps[:, 1], 1e-5) * 0.5) <= 4 * TOL[torch.bfloat16]
