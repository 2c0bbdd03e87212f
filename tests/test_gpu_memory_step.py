"""Decode steps of the matrix memory (GPU): the kernel for one token a request against the walk token by token, which the float32 set takes
for the same float32 inputs."""
import pytest
import torch

from spite_b200.engine.batch import Segment, build_step_batch
from spite_b200.kernels.cuda import CudaKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dim,vdim", [(64, 32), (128, 36), (128, 256), (256, 100), (256, 512), (32, 64), (128, 30)])
@pytest.mark.parametrize("slots", [[3], [2, 0, 1, 5, 4], [1, 2, 1, 1], list(range(40))])
def test_one_token_as_the_walk(dim, vdim, slots):
    """Sizes with a kernel of their own and those that the walk keeps; columns that fill no block; padding rows (the first row's slot again),
    which leave the state alone; states that start at zero beside used ones.  Both add up `dim` products in float32 in different orders:
    at most dim * 2^-24 of the sum of magnitudes, 1.6e-5 at 256, and the same of the denominator."""
    H, n = 3, len(slots)
    g = torch.Generator(device=DEV).manual_seed(dim + vdim + n)
    width = 2 * H * dim + H * vdim + 2 * H
    proj = torch.randn((n, width), generator=g, device=DEV)
    at = [0, H * dim, 2 * H * dim, 2 * H * dim + H * vdim, 2 * H * dim + H * vdim + H]
    first = torch.randn((max(slots) + 1, H, CudaKernels.mlstm_state_size(dim, vdim)), generator=g, device=DEV) * 0.3
    used = first[:, :, dim * vdim:]                          # the copies of (n, m) are one per 32 columns, all alike
    step = -(-(dim + 1) // 4) * 4
    for b in range(-(-vdim // 32)):
        used[:, :, b * step:(b + 1) * step] = used[:, :, :step].clone()
    first[0] = 0.0
    batch = build_step_batch([Segment(i, s, 9, 1, i, False) for i, s in enumerate(slots)], [[0]] * n, [[]] * n, [], DEV)
    bias = [torch.randn(H, generator=g, device=DEV) for _ in range(2)]
    got = []
    for dtype in (torch.bfloat16, torch.float32):
        ks, state, out = CudaKernels(dtype, DEV), first.clone(), torch.full((n, H * vdim), 7.0, device=DEV)
        for _ in range(2):
            ks.mlstm_scan(proj, out, batch, state, heads=H, dim=dim, vdim=vdim, gate_cap=6.0, q_scale=dim ** -0.5, columns=at, i_bias=bias[0],
                          f_bias=bias[1])
        torch.cuda.synchronize()
        got.append((out, state))
    for a, b, what in zip(*got, ("outputs", "states")):
        assert torch.isfinite(a).all() and float((a - b).abs().max()) <= 3.2e-5 * float(b.abs().max()), what
    padding = [i for i, s in enumerate(slots) if i and s == slots[0]]
    assert not padding or float(got[0][0][padding].abs().max()) == 0.0
