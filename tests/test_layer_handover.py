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
