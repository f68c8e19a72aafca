"""The norms between sublayers at the sizes where a launch changes its form: few rows (up to two an SM) and many, rows
that one, two or four vectors a thread hold, widths that leave threads without a vector.  Each against float64.

A row's sum of squares has W terms added in pieces: each thread its own few, then 32 lanes, then the warps, so under
W / 128 + 40 roundings of 2^-24 relative; a result has a few more.  The bounds are 64 + W / 128 roundings, and half a
unit of bfloat16 (2^-9) for outputs in that type."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from janus_b200.kernels import ops as o
    return o


def rnd(*shape, seed=0, s=1.0, mean=0.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * s + mean).to(DEV)


def check(got, want, W):
    tol = (64 + W / 128) * 2.0 ** -24 + (2.0 ** -8 if got.dtype == torch.bfloat16 else 0.0)
    want = want.double()
    assert float(((got.double() - want).abs() / (want.abs() + want.abs().mean())).max()) <= tol


ROWS = [1, 296, 297]


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("W", [1020, 1024, 2048, 2052, 4096, 4100, 8192, 8196])
def test_rmsnorm_and_sublayer(ops, rows, W):
    x, gamma, eps = rnd(rows, W), rnd(W, seed=1, s=0.1, mean=1.0).to(torch.bfloat16), 1e-5
    clear, out = rnd(777 * 4), torch.empty(rows, W, dtype=torch.bfloat16, device=DEV)
    pick = torch.arange(rows - 1, -1, -1, dtype=torch.int32, device=DEV)
    ops.rmsnorm(x, gamma, eps, out, row_index=pick, clear=clear)
    unit = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + eps) * gamma.double()
    check(out, unit[pick.long()], W)
    assert not bool(clear.any())
    y, residual, clear = x.clone(), rnd(rows, W, seed=2), rnd(64)
    want = residual.double() + 0.7 * unit
    ops.sublayer_norm_add(y, gamma, eps, 0.7, residual, out, clear=clear)
    check(residual, want, W)
    check(out, want, W)
    assert not bool(y.any()) and not bool(clear.any())


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("W", [508, 512, 2048, 2052, 4096, 4100])
@pytest.mark.parametrize("S", [2, 3, 4, 5])
def test_streams(ops, rows, W, S):
    x, y, eps = rnd(rows, S * W), rnd(rows, W, seed=1), 1e-5
    mix, into, read, gamma = rnd(S, S, seed=2), rnd(S, seed=3), rnd(S, seed=4), rnd(W, seed=5, s=0.1, mean=1.0).to(torch.bfloat16)
    out, clear2 = torch.empty(rows, W, dtype=torch.bfloat16, device=DEV), rnd(1000)
    old = x.double().view(rows, S, W)

    def normed(streams, weights):
        u = torch.einsum("s,rsw->rw", weights.double(), streams)
        return u / torch.sqrt((u ** 2).mean(-1, keepdim=True) + eps) * gamma.double()
    ops.streams_rmsnorm(x, S, read, gamma, eps, out, clear=y.clone(), clear2=clear2)
    check(out, normed(old, read), W)
    pick = torch.arange(rows - 1, -1, -1, dtype=torch.int32, device=DEV)
    ops.streams_rmsnorm(x, S, None, gamma, eps, out, row_index=pick)
    check(out, normed(old, torch.ones(S, device=DEV))[pick.long()], W)
    new = torch.einsum("st,rsw->rtw", mix.double(), old) + into.double()[None, :, None] * y.double()[:, None, :]
    ops.streams_mix_rmsnorm(x, y, mix, into, read, S, gamma, eps, out, clear2=clear2)
    size = torch.einsum("st,rsw->rtw", mix.double().abs(), old.abs()) + (into.double()[None, :, None] * y.double()[:, None, :]).abs()
    assert bool(((x.double().view(rows, S, W) - new).abs() <= 16 * 2.0 ** -24 * size + 1e-6).all())
    check(out, normed(new, read), W)
    assert not bool(clear2.any()) and not bool(y.any())


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("W", [508, 512, 1000, 2048, 2052, 4096, 4100])
@pytest.mark.parametrize("form", ["norm", "one", "two", "sum"])
def test_join(ops, rows, W, form):
    r, ya, yb, eps = rnd(rows, W), rnd(rows, W, seed=1), rnd(rows, W, seed=2), 1e-5
    wa, wb, scale, gamma, extra = (rnd(W, seed=i, s=0.1, mean=1.0) for i in (3, 4, 5, 6, 7))
    extra = rnd(rows, W, seed=8)
    unit = lambda t: t / torch.sqrt((t ** 2).mean(-1, keepdim=True) + eps)                  # noqa: E731
    out, clear, clear2 = torch.empty(rows, W, dtype=torch.bfloat16, device=DEV), rnd(3000), rnd(12)
    want, kw = r.double(), {}
    if form == "one":
        want, kw = want + scale.double() * ya.double() + extra.double(), dict(ya=ya, scale=scale, extra=extra)
    elif form == "two":
        want = want + 0.5 * (unit(ya.double()) * wa.double() + unit(yb.double()) * wb.double())
        kw = dict(ya=ya, yb=yb, wa=wa, wb=wb, mult=0.5)
    elif form == "sum":
        want, kw = want + 0.8 * ya.double() + 0.9 * yb.double(), dict(ya=ya, yb=yb, mult=0.8, mult_b=0.9)
    center = form != "sum"
    ops.join_norm(r, gamma=gamma, eps=eps, center=center, x_out=out, clear=clear, clear2=clear2, **kw)
    check(r, want, W)
    base = want - want.mean(-1, keepdim=True) if center else want
    check(out, unit(base) * gamma.double(), W)
    assert not bool(clear.any()) and not bool(clear2.any())
    if form != "norm":
        assert not bool(ya.any())
    if form in ("two", "sum"):
        assert not bool(yb.any())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W", [1024, 2048, 2052, 4096, 4100, 8192, 8200])
def test_a_row_is_the_same_alone_and_among_many(ops, W, dtype):
    """Bit for bit, whatever form the number of rows selects: a row alone, among 148 or 296 (few) and among 300 (many)."""
    many, eps = 300, 1e-5
    x, y, res, gate = rnd(many, W), rnd(many, W, seed=1), rnd(many, W, seed=2), rnd(many, W, seed=3)
    streams, mix, into = rnd(many, 2 * W, seed=4), rnd(2, 2, seed=5), rnd(2, seed=6)
    gamma, wa, wb = (rnd(W, seed=i, s=0.1, mean=1.0) for i in (7, 8, 9))

    def norms(rows):
        at = slice(many - rows, many)
        made = []

        def out():
            made.append(torch.empty(rows, W, dtype=dtype, device=DEV))
            return made[-1]
        ops.rmsnorm(x[at].clone(), gamma, eps, out())
        r = res[at].clone()
        ops.sublayer_norm_add(y[at].clone(), gamma, eps, 0.7, r, out())
        made.append(r)
        ops.streams_rmsnorm(streams[at].clone(), 2, into, gamma, eps, out())
        s = streams[at].clone()
        ops.streams_mix_rmsnorm(s, y[at].clone(), mix, into, into, 2, gamma, eps, out())
        made.append(s)
        for center in (True, False):
            r = res[at].clone()
            ops.join_norm(r, gamma=gamma, eps=eps, center=center, x_out=out(), ya=y[at].clone(), yb=x[at].clone(), wa=wa, wb=wb, mult=0.5)
            made.append(r)
        ops.gated_rmsnorm(x[at].clone(), gamma, gate[at].clone(), eps, out())
        ops.gated_group_rmsnorm(x[at].clone(), gate[at].clone(), gamma, eps, 1, out())
        if W % 8 == 0:
            ops.gated_group_rmsnorm(x[at].clone(), gate[at].clone(), gamma, eps, 2, out())
        return [m[-1] for m in made]
    want = norms(many)
    for rows in (1, 100, 148, 296, 297):
        assert [i for i, (a, b) in enumerate(zip(norms(rows), want)) if not torch.equal(a, b)] == [], rows


def test_float32_logits_do_not_depend_on_the_step(ops):
    """The 32-bit engine, bit for bit: a prompt of 400 tokens in one step, cut at 100, token after token at its end, and with
    another sequence's tokens in the step."""
    import janus_b200
    from janus_b200.engine import StepEntry
    config = dict(architectures=["LlamaForCausalLM"], hidden_size=1024, num_hidden_layers=2, num_attention_heads=8,
                  num_key_value_heads=2, head_dim=128, intermediate_size=2048, vocab_size=1000, max_position_embeddings=1024,
                  rms_norm_eps=1e-5, rope_theta=10000.0, tie_word_embeddings=False)
    model = janus_b200.load_random(config, seed=3, dtype="float32", max_tokens=2048)
    g = torch.Generator().manual_seed(0)
    tokens, other = (torch.randint(0, 1000, (n,), generator=g).tolist() for n in (400, 77))

    def logits(cuts, beside=None):
        slots, at, rows = [model.alloc_slot(), model.alloc_slot()], 0, []
        for end in cuts + [400]:
            entries = [StepEntry(slots[0], tokens[at:end], range(end - at))]
            if beside is not None and at == 0:
                entries.insert(0, StepEntry(slots[1], beside, (0,)))
            rows.append(model.step(entries)[-(end - at):].clone())
            at = end
        for s in slots:
            model.free_slot(s)
        return torch.cat(rows)
    want = logits([])
    for cuts, beside in (([100], None), ([296], None), ([397, 398, 399], None), ([100], other), ([], other)):
        assert torch.equal(logits(cuts, beside), want), cuts
