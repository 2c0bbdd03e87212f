"""What a layer begins with, made by the last kernel of the layer before: the same logits as of the layers one by one (which a tap asks
for)."""
import pytest
import torch

import gapevik_helpers
import helpers as H
import paposun_helpers
from reference_kernels import TorchReferenceKernels
from spite_b200.engine import Engine, Model


@pytest.mark.parametrize("helper,name", [(paposun_helpers, "K"), (paposun_helpers, "M"), (gapevik_helpers, "A"), (gapevik_helpers, "C")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_same_logits_as_layer_by_layer(helper, name, dtype, tmp_path):
    model = Model.from_folder(helper.write_model(tmp_path, name), dtype=str(dtype).split(".")[1], device="cpu", kernels=TorchReferenceKernels(dtype, "cpu"))
    steps = H.steps_last_decoded({f"r{i}": H.random_tokens(model.plan.vocab_size, n, 40 + i) for i, n in enumerate((9, 1, 20))}, 4)
    got = []
    for tap in (None, lambda i, h: None):
        model.layer_tap = tap
        got.append(H.run_steps(Engine(model, cache_tokens=192, page_size=16, max_requests=4), steps))
    assert got[0].keys() == got[1].keys() and len(got[0]) == 30
    assert all(torch.equal(logits, got[1][at]) for at, logits in got[0].items())
    if helper is paposun_helpers or dtype == torch.bfloat16:       # (float32 products of the other kind read the stream in place)
        order = [model.blocks[c.layer] for c in model.plan.order if hasattr(c, "layer")]
        assert any(a.leaves(b.entry()) for a, b in zip(order, order[1:]))


@pytest.mark.parametrize("helper,name", [(paposun_helpers, "K"), (gapevik_helpers, "A")])
@pytest.mark.parametrize("wrap", ["blocks", "norms"])
def test_wrapped_parts_are_called(helper, name, wrap, tmp_path):
    """A program that wraps a block's or a norm's forward sees every call of it, with the arguments of a layer by itself."""
    model = Model.from_folder(helper.write_model(tmp_path, name), dtype="bfloat16", device="cpu", kernels=TorchReferenceKernels(torch.bfloat16, "cpu"))
    steps = H.steps_last_decoded({"r": H.random_tokens(model.plan.vocab_size, 9, 40)}, 3)
    plain, calls = H.run_steps(Engine(model, cache_tokens=192, page_size=16, max_requests=4), steps), []

    def watch(part):
        forward = part.forward
        if wrap == "blocks":
            part.forward = lambda h, batch, cache: (calls.append(part), forward(h, batch, cache))[1]
        else:
            part.forward = lambda h, out, rows=None: (calls.append(part), forward(h, out, rows))[1]
    parts = model.blocks if wrap == "blocks" else [b.mixer_norm for b in model.blocks if hasattr(b, "mixer_norm") and b.kind == "sandwich_residual"]
    for part in parts:
        watch(part)
    got = H.run_steps(Engine(model, cache_tokens=192, page_size=16, max_requests=4), steps)
    runs = [c.layer for c in model.plan.order if hasattr(c, "layer")] if wrap == "blocks" else \
        [c.layer for c in model.plan.order if hasattr(c, "layer") and model.blocks[c.layer].kind == "sandwich_residual"]
    assert len(calls) == len(steps) * len(runs)
    assert all(torch.equal(logits, got[at]) for at, logits in plain.items())
