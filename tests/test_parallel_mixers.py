"""Two mixers side by side whose projections are one product: widths whose buffers are no whole vectors."""
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
