"""Two mixers side by side whose projections are one product: widths whose buffers are no whole vectors, and either
branch on either side."""
import pytest
import torch

from helpers import random_tokens, rel_err
from test_mugedra import folder, layer, left, load, plain_logits, right, tol_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("width", [1025, 2051])
def test_a_shared_product_is_cleared_whatever_the_width(tmp_path, width):
    """An odd width and an odd number of tokens: the branches' buffers end off a 16-byte boundary, so the product whose slices of
    K meet by adds has a buffer of its own.  All scratch comes filled with NaN, in a first pass and in later ones."""
    from janus_b200.engine import StepEntry
    cfg = dict(architecture="Mugedra", vocab=96, width=width, norm=dict(eps=1e-5),
               layers=[layer(left(2, 1, 16, 16, 0.25, mask=40, rot=(8, 100.0)), right(2, 2, 16, 16, 3)),
                       layer(left(4, 2, 8, 16, 0.3), right(2, 1, 8, 24, 2))])
    d, w = folder(tmp_path, cfg, 21)
    model = load(d, "bfloat16")
    assert all(place.mixer.proj.meets_by_adds(n, torch.float32) for place in model.engine.model.layers for n in (1, 3))
    ids = random_tokens(7, cfg["vocab"], 5)
    ref = plain_logits(cfg, w, ids)
    for _ in range(3):
        slot, got, at = model.alloc_slot(), [], 0
        for n in (3, 1, 1, 1, 1):
            for buf in model.engine.workspace._buffers.values():
                if buf.is_floating_point():
                    buf.fill_(float("nan"))
            got.append(model.step([StepEntry(slot, ids[at:at + n], range(n))]).cpu())
            at += n
        model.free_slot(slot)
        assert rel_err(torch.cat(got), ref) < tol_for("bfloat16")
    model.check()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_either_branch_on_either_side(tmp_path, monkeypatch, dtype):
    """Attention on the right, the recurrence on the left: the sum of both is the same model."""
    from janus_b200.engine import StepEntry
    from janus_b200.models import mugedra
    from janus_b200.parts.base import PartSpec
    made = mugedra._mixer_spec
    other = {"left": "right", "right": "left"}

    def swapped(config, i):
        spec = made(config, i)
        params = dict(spec.params, left=spec.params["right"], right=spec.params["left"])
        weights = {other[n[:n.index("_out")]] + "_out" if n.endswith("_out") else other[n.split(".", 1)[0]] + "." + n.split(".", 1)[1]: t
                   for n, t in spec.weights.items()}
        return PartSpec(spec.kind, params, weights=weights)

    monkeypatch.setattr(mugedra, "_mixer_spec", swapped)
    cfg = dict(architecture="Mugedra", vocab=96, width=64, norm=dict(eps=1e-5),
               layers=[layer(left(4, 2, 16, 24, 0.3, softcap=4.0, mask=37, rot=(8, 1000.0)), right(4, 2, 8, 16, 3)),
                       layer(left(2, 1, 32, 16, 0.2), right(2, 2, 16, 8, 4))])
    d, w = folder(tmp_path, cfg, 22)
    model = load(d, dtype)
    kinds = [type(b).__name__ for b in model.engine.model.layers[0].mixer.branches.values()]
    assert kinds == ["GatedDeltaRule", "CappedAttention"]
    ids = random_tokens(75, cfg["vocab"], 6)
    slot = model.alloc_slot()
    got = [model.step([StepEntry(slot, ids[:70], range(70))]).cpu()]
    got += [model.step([StepEntry(slot, [t], [0])]).cpu() for t in ids[70:]]
    assert rel_err(torch.cat(got), plain_logits(cfg, w, ids)) < tol_for(dtype)
    model.check()
