"""Gains, taps and biases that the kernel right before makes (GPU): the kernels of a step overlap, so a kernel may read them only once that one has
ended.  Each is made by a product that takes its time and read by the next launch; the same calls with a wait in between give the bits
that must come out."""
import pytest
import torch

from spite_b200.engine.batch import Segment, build_step_batch
from spite_b200.kernels.cuda import CudaKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d", [256, 2048, 5120, 8192])
@pytest.mark.parametrize("what", ["norm", "residual gain", "residual next gain", "taps 4", "taps 7", "taps 4 bias"])
def test_made_by_the_kernel_before(what, d):
    ks, K, M = CudaKernels(torch.bfloat16, DEV), 8192, 12
    g = torch.Generator(device=DEV).manual_seed(d + len(what))
    rnd = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    taps = int(what.split()[1]) if what.startswith("taps") else 1
    n = d if what.endswith("bias") else d * taps
    w = rnd(n, K).to(torch.bfloat16) / 64
    x, y, rest = rnd(M, d), rnd(M, d), rnd(d * taps)
    batch = build_step_batch([Segment(0, 0, 0, M, 0, True)], [[0] * M], [[]], [], DEV)

    def passes(wait):
        made, results = torch.full((1, n), 7.0, device=DEV), []
        for i in range(8):
            source = torch.randn((1, K), generator=torch.Generator(device=DEV).manual_seed(i), device=DEV).to(torch.bfloat16)
            h, state, out = x.clone(), torch.zeros((1, max(1, (taps - 1) * d)), device=DEV), torch.empty((M, d), dtype=torch.bfloat16, device=DEV)
            ks.linear(source, w, made)
            if wait:
                torch.cuda.synchronize()
            if what == "norm":
                ks.rms_norm(h, made[0], 1e-5, out)
            elif what == "residual gain":
                ks.rms_norm_residual(y, made[0], 1e-5, 0.5, h, next_gain=rest, next_out=out)
            elif what == "residual next gain":
                ks.rms_norm_residual(y, rest, 1e-5, 0.5, h, next_gain=made[0], next_out=out)
            elif what.endswith("bias"):
                ks.short_conv(x, rest.view(d, taps), out, batch, state, channels=d, activation="silu", bias=made[0])
            else:
                ks.short_conv(x, made.view(d, taps), out, batch, state, channels=d, activation="silu")
            results += [h, out, state]
        torch.cuda.synchronize()
        return results
    for a, b in zip(passes(False), passes(True)):
        assert torch.equal(a, b)
