"""The state space's walk in chunks with 64 value columns a block (GPU), which it takes where all blocks are then resident at once: the same bits
as with 32, which the same segments take one by one."""
import pytest
import torch

from spite_b200.engine.batch import Segment, build_step_batch
from spite_b200.kernels.cuda import CudaKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,lengths", [
    (60, 60, 64, 64, [97, 33, 300, 64]),       # 240 blocks of 64 columns (480 of 32)
    (74, 1, 48, 64, [40, 129, 32, 65]),        # 296: all that are resident at once; keys that fill no tile
    (75, 1, 64, 64, [40, 129, 32, 65]),        # one head more: 32 columns
    (16, 4, 64, 128, [70, 35, 200, 96, 33, 64, 41, 500]),
    (120, 8, 20, 40, [100, 57])])              # 240 blocks whose second half has 8 columns
def test_columns_of_a_block(heads, kv_heads, dim, vdim, lengths):
    ks, g = CudaKernels(torch.bfloat16, DEV), torch.Generator(device=DEV).manual_seed(heads + vdim)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    M = sum(lengths)
    q, k, v, step = rnd(M, kv_heads * dim) * 0.3, rnd(M, kv_heads * dim) * 0.3, rnd(M, heads * vdim), rnd(M, heads)
    a_log, dt_bias, skip = rnd(heads) * 0.3, rnd(heads), rnd(heads)
    state = rnd(len(lengths), heads * ks.scan_state_size(dim, vdim)) * 0.1

    def walk(lengths, slots, rows):
        segs, at = [], 0
        for i, n in enumerate(lengths):
            segs.append(Segment(i, slots[i], 0, n, at, False))
            at += n
        batch = build_step_batch(segs, [[0] * n for n in lengths], [[] for _ in lengths], [], DEV)
        out = torch.full((at, heads * vdim), float("nan"), device=DEV)
        parts = [(t[rows].contiguous(), 0) for t in (q, k, v, step)]
        ks.state_space_scan(*parts, out, batch, states, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, a_log=a_log, dt_bias=dt_bias, skip=skip,
                            chunked=True)
        return out
    states = state.clone()
    together, after = walk(lengths, list(range(len(lengths))), slice(0, M)), states
    states, at = state.clone(), 0
    for i, n in enumerate(lengths):
        assert torch.equal(walk([n], [i], slice(at, at + n)), together[at:at + n])
        at += n
    torch.cuda.synchronize()
    assert torch.equal(states, after) and torch.isfinite(together).all() and ks.errors() == {}
