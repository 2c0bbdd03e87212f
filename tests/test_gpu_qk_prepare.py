"""Queries and keys on their way to the attention (GPU): the kernel that moves 16-byte words against the one that moves pairs, which takes the
same rows when they lie two elements apart from a multiple of eight."""
import pytest
import torch

from spite_b200.cache import LayerCache
from spite_b200.kernels.cuda import CudaKernels
from spite_b200.parts.base import QkNorm, Rotation
from test_gpu_kernels import make_batch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("specs", [[(4000, 1)], [(0, 5), (77, 1)], [(130, 255)], [(63, 256)], [(1000, 200), (0, 130), (9, 1)]])
@pytest.mark.parametrize("nq,nkv,hd,pairing,rot,norm,rest", [
    (8, 2, 128, "neighbours", 128, "after", ""), (5, 1, 128, "neighbours", 50, "before", "gain"), (40, 8, 128, "halves", 128, "after", "gain bias"),
    (6, 6, 64, "halves", 32, "before", "gain temperature"), (3, 1, 64, "neighbours", 2, None, "bias gates"), (12, 2, 64, "halves", 16, "after", "narrow"),
    (7, 7, 128, None, 0, "after", "temperature gates"), (9, 3, 128, "halves", 64, None, "q_only bias"), (4, 4, 64, None, 0, None, "read")])
def test_words_as_pairs(specs, nq, nkv, hd, pairing, rot, norm, rest):
    ks, P = CudaKernels(torch.bfloat16, DEV), 64
    n_pages = sum(-(-(s + n) // P) for s, n in specs) + 2
    batch, _ = make_batch(specs, P, n_pages, 5, DEV)
    M, g = batch.n_tokens, torch.Generator(device=DEV).manual_seed(nq * 100 + hd + rot)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    cols = (nq + (0 if "q_only" in rest else 2 * nkv)) * hd
    wide = rnd(M, cols + 48).to(torch.bfloat16)              # (48: the gates' columns, at the most)
    rotation = None if pairing is None else Rotation(1e4 ** (-torch.arange(rot // 2, device=DEV) / (rot / 2.0)), pairing, rot, 1.25)
    gain = "gain" in rest
    qk_norm = None if norm is None else QkNorm(1e-5, norm == "before", rnd(hd) if gain else None, rnd(hd) if gain else None)
    got = []
    for pad in (0, 2):
        qkv = torch.empty((M, cols + 48 + pad), dtype=torch.bfloat16, device=DEV)
        qkv[:, :cols + 48] = wide
        q, kv = torch.full((M, nq * hd), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((2, n_pages, nkv, P, hd), 7.0, dtype=torch.bfloat16, device=DEV)
        gates = torch.zeros((M, nq), device=DEV) if "gates" in rest else None
        g2 = torch.Generator(device=DEV).manual_seed(3)
        ks.qk_prepare(qkv, q, batch, LayerCache(0, kv, None, P, not ("q_only" in rest or "read" in rest)), num_heads=nq, rotation=rotation,
                      qk_norm=qk_norm, temperature=(100, 0.1) if "temperature" in rest else None, gates_out=gates, q_only="q_only" in rest,
                      bias=torch.randn(cols, generator=g2, device=DEV) if "bias" in rest else None, norm_dim=hd - 3 if "narrow" in rest else None)
        torch.cuda.synchronize()
        got.append([q.float(), kv.float()] + ([gates] if gates is not None else []))
    for a, b, what in zip(*got, ("queries", "cache", "gates")):
        # a norm's sum is added in another order (2^-22 of it), so a rounding to bfloat16 may go the other way: one unit, 2^-8 of the element;
        # where a rotation's two products cancel the difference is 2^-22 of the products
        assert float(((a - b).abs() - 2.0 ** -7 * b.abs() - 2e-6).max()) <= 0.0, what
        assert float((a != b).float().mean()) < 0.02, what
