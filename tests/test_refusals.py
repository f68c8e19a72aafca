"""Calls that would read or write past their tensors, or ask for more than a launch can have, are refused before anything is
launched (no GPU: the faces of the kernels on host tensors, and the C functions themselves)."""
import pytest
import torch

from janus_b200.kernels import ops

BAD_SIZE = 10001


@pytest.fixture
def launched(monkeypatch):
    """Faces without a device: the arguments of the C functions that were reached."""
    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append((name, a)) or 0

    monkeypatch.setattr(ops, "_lib", lambda *a: Lib())
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    with ops.unchecked():
        yield calls


def head_step(kind, T=2, H=4, G=None, d=8, e=8, rank=6, state=None, m_off=None, raw_cols=None, cols=None, ab=None):
    G = H if G is None else G
    memory, channel = kind == "memory", kind == "channel"
    m_off = (H * d * (e + 1) if memory else 0) if m_off is None else m_off
    state = (H * d * (e + memory) + (H if memory else 0) if state is None else state)
    low = rank if channel else 2 * H
    q, k, v = (0, G * d, 2 * G * d) if cols is None else cols
    z = lambda *s: torch.zeros(*s)     # noqa: E731
    rows, raw = z(T, 2 * G * d + H * e), z(T, low if raw_cols is None else raw_cols)
    a, b = (0, 0 if channel else H) if ab is None else ab
    ints = lambda n: torch.zeros(n, dtype=torch.int32)   # noqa: E731
    ops.head_step(kind, rows, q, k, v, 1.0, raw, a, b, z(rank, H * d) if channel else z(H), z(H * d) if channel else z(H), 1.0,
                  z(T, state), z(T, H * e), z(e), 1e-5, z(T, H * e), ints(T + 1), ints(T), H, G, d, e, m_off=m_off)


@pytest.mark.parametrize("kind", ["delta", "memory", "channel"])
def test_head_step_takes_what_fits(launched, kind):
    head_step(kind)
    if kind == "delta":
        head_step(kind, G=2)
    assert launched


@pytest.mark.parametrize("kind, how", [
    ("memory", dict(m_off=4 * 8 * 9 + 1)), ("memory", dict(m_off=4 * 8 * 9 + 4)), ("memory", dict(state=4 * 8 * 9 + 3)),
    ("delta", dict(state=255)), ("delta", dict(raw_cols=7)), ("memory", dict(raw_cols=7)), ("channel", dict(raw_cols=5)),
    ("delta", dict(ab=(5, 0))), ("memory", dict(ab=(0, 5))), ("channel", dict(ab=(1, 0))), ("memory", dict(G=2)), ("channel", dict(G=1)),
    ("delta", dict(cols=(65, 32, 64))), ("delta", dict(cols=(0, 65, 64))), ("delta", dict(cols=(0, 32, 65)))])
def test_head_step_refuses(launched, kind, how):
    """Maxima behind the slot's row, gates' columns behind the matrix, fewer key heads than the kind reads."""
    with pytest.raises(ops.KernelError):
        head_step(kind, **how)
    assert not launched


@pytest.mark.parametrize("kind, changed", [
    (1, dict(m_off=292)), (1, dict(m_off=289)), (1, dict(G=2)), (2, dict(G=2)), (2, dict(rank=9)), (0, dict(col_a=5)), (1, dict(col_b=5)),
    (0, dict(slot_stride=252)), (0, dict(q_col=65)), (0, dict(k_col=-4)), (0, dict(v_col=68)), (2, dict(col_a=-1))])
def test_the_c_entry_of_head_step_refuses_them_too(kind, changed):
    """Four heads of 8 x 8 in rows of 96 and gates' arguments in rows of 8; nothing is launched, so no pointer is followed."""
    a = dict(kind=kind, rows=0, ld=96, q_col=0, k_col=32, v_col=64, q_scale=1.0, raw=0, ld_raw=8, col_a=0, col_b=4, p0=0, p1=0, scalar=1.0,
             rank=8, state=0, slot_stride=292, state_off=0, m_off=288, gate=0, ld_gate=32, weight=0, w_stride=0, act=0, eps=1e-5, out=0,
             out_dtype=0, q_start=0, seq_slot=0, n_seqs=1, H=4, G=4, d=8, e=8, stream=0)
    assert set(changed) <= set(a)
    a.update(changed)
    assert ops._lib("head_step").jb_head_step(*a.values()) == BAD_SIZE


def test_a_router_of_more_rows_than_a_launch_holds():
    """3 numbers a row lie in shared memory, of which a launch has 48 KB: 8,192 rows of 8 numbers go in two launches."""
    from janus_b200.parts.routed import RoutedExperts
    part = RoutedExperts(8, 8, 8192, 2, dtype=torch.bfloat16, device=torch.device("cpu"))
    assert not part.route_in_one
    assert ops._lib("routed").jb_route_tokens(0, 0, 8, 8192, 0, 8192, 2, 0, 0, 1, 0, 0, 0, 0, 1.0, 0, 1, 0) == BAD_SIZE
    assert ops._lib("routed").jb_route_tokens(0, 0, 8, 4097, 0, 4097, 2, 0, 0, 1, 0, 0, 0, 0, 1.0, 0, 1, 0) == BAD_SIZE


@pytest.mark.parametrize("rows, width, one", [(8, 2048, True), (16, 2048, True), (24, 2048, True), (9, 4096, True), (12, 4096, True), (8, 264, True),
                                              (24, 8, True), (25, 8, False), (13, 4096, False), (8, 8192, False), (64, 512, False)])
def test_which_routers_choose_in_the_product_s_launch(rows, width, one):
    """On both sides of the lines in rows and in numbers; a shared expert's gate is a row too."""
    from janus_b200.parts.routed import RoutedExperts
    for gate in (False, True):
        part = RoutedExperts(width, 8, rows - gate, 2, shared_size=8 if gate else None, shared_gate=gate, dtype=torch.bfloat16,
                             device=torch.device("cpu"))
        assert part.route_in_one is one


@pytest.mark.parametrize("kind, n, heads, dim, vdim, one", [
    ("delta", 256, 64, 32, 32, True), ("channel", 1, 16, 128, 128, True), ("channel", 96, 16, 128, 128, True), ("channel", 97, 16, 128, 128, False),
    ("channel", 64, 32, 64, 64, False), ("memory", 24, 64, 32, 64, True), ("memory", 25, 64, 32, 64, False), ("memory", 256, 32, 128, 64, True),
    ("memory", 256, 32, 64, 128, True), ("memory", 256, 32, 64, 124, False)])
def test_which_single_token_steps_are_one_launch(kind, n, heads, dim, vdim, one):
    assert ops.head_step_pays(kind, n, heads, dim, vdim) is one


@pytest.mark.parametrize("T, top, experts, F, W, tiles", [
    (1, 2, 8, 4096, 2048, True), (64, 2, 8, 4096, 2048, True), (2, 2, 8, 7168, 4096, True), (16, 2, 8, 7168, 4096, True), (1, 6, 64, 1408, 2048, True),
    (64, 8, 128, 768, 2048, True), (32, 8, 256, 512, 1024, True), (8, 10, 512, 512, 2048, True), (64, 16, 16, 512, 1024, True),
    (1, 1, 512, 128, 256, True), (1, 2, 8, 1536, 1024, False), (64, 2, 8, 1536, 1024, False), (1, 1, 1, 128, 128, False),
    (64, 2, 8, 128, 128, False), (16, 1, 4, 1024, 1024, False), (32, 4, 40, 256, 384, False), (8, 2, 16, 1024, 2048, False)])
def test_which_experts_stream_their_tiles(T, top, experts, F, W, tiles):
    """Sizes whose forms were measured more than 3 % apart, or that are a model's own."""
    assert ops.experts_stream_pays(T, top, experts, F, W) is tiles


@pytest.mark.parametrize("heads, dim, vdim, lens, chunks", [
    (16, 128, 128, [64], True), (16, 128, 128, [300, 300], True), (16, 128, 128, [400] * 8, True), (32, 128, 128, [1000, 1000], True),
    (32, 128, 128, [55] * 32, False), (16, 128, 128, [55] * 32, False), (16, 96, 64, [55] * 32, False), (16, 128, 128, [64] * 16, True),
    (16, 96, 64, [700] * 4, False), (16, 96, 64, [275] * 8, True), (16, 128, 128, [1000], False), (16, 64, 64, [55] * 32, False)])
def test_which_prompts_of_channel_decays_go_by_chunks(heads, dim, vdim, lens, chunks):
    """On both sides of the lines in blocks, tokens and width of the values."""
    assert ops.state_chunks_pay("channel", len(lens), heads, dim, vdim, max(lens), sum(lens)) is chunks
