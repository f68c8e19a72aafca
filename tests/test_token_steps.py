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
