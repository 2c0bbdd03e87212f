"""The short convolution over segments of several tokens (GPU): the kernel of four columns a thread, at every number of taps, against the one of
a column a thread, which takes the same rows when the slots' state lies off a 16-byte boundary.  The sums are the same, term by term."""
import pytest
import torch

from spite_b200.engine.batch import Segment, build_step_batch
from spite_b200.kernels.cuda import CudaKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps", range(1, 9))
def test_every_number_of_taps(taps, dtype):
    ks, channels, extra, slots = CudaKernels(torch.bfloat16, DEV), 520, 8, [2, 0, 3]
    g = torch.Generator(device=DEV).manual_seed(taps)
    w, bias = torch.randn((channels, taps), generator=g, device=DEV), torch.randn(channels, generator=g, device=DEV)
    n_state = (taps - 1) * channels
    states = [torch.zeros((4, n_state + 4), device=DEV) for _ in range(2)]
    for counts in ([9, 20, 4], [1, 5, 33], [8, 2, 7]):
        segs, M = [], 0
        for s, n in enumerate(counts):
            segs.append(Segment(s, slots[s], 0, n, M, False))
            M += n
        batch = build_step_batch(segs, [[0] * n for n in counts], [[] for _ in counts], [], DEV)
        x, outs = torch.randn((M, channels + extra), generator=g, device=DEV), []
        for offset, state in enumerate(states):
            outs.append(torch.full((M, channels + extra), 7.0, dtype=dtype, device=DEV))
            ks.short_conv(x, w, outs[-1], batch, state, channels=channels, activation="silu", state_offset=offset, bias=bias)
        assert torch.equal(*outs)
        assert torch.equal(states[0][:, :n_state], states[1][:, 1:n_state + 1])
    assert not states[0][1].any() and not states[0][:, n_state:].any()
