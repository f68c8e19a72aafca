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


@pytest.mark.parametrize("T, W, E", [(16, 1184, 8), (16, 1200, 8), (1, 2048, 4), (3, 4736, 4)])
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
