"""A model's factor of the logits: multiplied in by the head's product up to a number of rows, by a pass over the logits beyond it.  Both are
the stored sum times the factor, the same number."""
import pytest
import torch

import helpers as H
import paposun_helpers
from reference_kernels import TorchReferenceKernels
from spite_b200.engine import Engine, Model


class Passes:
    """Counts the passes over the logits of a kernel set."""

    def __init__(self, kernels):
        self.kernels, self.passes = kernels, 0

    def __getattr__(self, name):
        if name == "transform_logits":
            self.passes += 1
        return getattr(self.kernels, name)


@pytest.mark.parametrize("most", [0, 1, 12, 13])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_beyond_the_limit(dtype, most, tmp_path, monkeypatch):
    """Steps of 13 rows and of one: with a limit of 12 the first takes the pass and the others do not."""
    folder, got = paposun_helpers.write_model(tmp_path, "K"), []
    for limit in (most, Model.scaled_logit_rows):
        monkeypatch.setattr(Model, "scaled_logit_rows", limit)
        kernels = Passes(TorchReferenceKernels(dtype, "cpu"))
        model = Model.from_folder(folder, dtype=str(dtype).split(".")[1], device="cpu", kernels=kernels)
        assert model.plan.logit_scale != 1.0
        steps = H.steps_last_decoded({"r": H.random_tokens(model.plan.vocab_size, 17, 3)}, 4)
        got.append((H.run_steps(Engine(model, cache_tokens=64, page_size=16, max_requests=2), steps), kernels.passes))
    assert [n for _, n in got] == [{0: 5, 1: 1, 12: 1, 13: 0}[most], 0] and len(got[0][0]) == 17
    assert all(torch.equal(row, got[1][0][at]) for at, row in got[0][0].items())


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 4, 16, 24, 33, 300, 5000])
@pytest.mark.parametrize("N,K", [(1000, 256), (70016, 128), (211, 72)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_product_gives_the_passes_bits(dtype, N, K, M):
    """Every kernel that a head's product may take, by rows, width and depth."""
    from spite_b200.kernels.cuda import CudaKernels
    if M * N > 1 << 26:
        M = (1 << 26) // N
    ks, g = CudaKernels(dtype, "cuda:0"), torch.Generator(device="cuda:0").manual_seed(M + N)
    x, w = (torch.randn(shape, generator=g, device="cuda:0").to(dtype) for shape in ((M, K), (N, K)))
    a, b = torch.empty((M, N), device="cuda:0"), torch.empty((M, N), device="cuda:0")
    ks.linear(x, w, a, row_scale=torch.full((M,), 0.3, device="cuda:0"))
    ks.linear(x, w, b)
    ks.transform_logits(b, scale=0.3)
    assert torch.equal(a, b) and ks.errors() == {}
