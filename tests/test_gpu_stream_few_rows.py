"""Decode products of one to sixteen rows as the kernel set cuts them: sums against float64, and token columns that nobody asks for (they hold
whatever lay in shared memory) kept out of the others."""
import pytest
import torch

from spite_b200.kernels.cuda import CudaKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K", [(40, 64), (129, 192), (1024, 4096), (2048, 2048), (4096, 1024)])
def test_few_rows_against_float64(N, K):
    """A float32 sum of K products: each of its at most K roundings is below 2^-24 of the sum of magnitudes."""
    ks = CudaKernels(torch.bfloat16, DEV)
    g = torch.Generator().manual_seed(N + K)
    w = torch.randn((N, K), generator=g).to(torch.bfloat16)
    w3 = torch.stack([w, w.roll(1, 0), w.roll(2, 0)]).to(DEV)
    before, calls = ks.launches_by_library["gemm_stream"], 0
    for M in (1, 2, 3, 5, 7, 8, 9, 12, 15, 16):
        # a product of 16 rows of NaN leaves NaN in every column of the shared memory that the next one finds
        ks.linear(torch.full((16, K), float("nan"), dtype=torch.bfloat16, device=DEV), w.to(DEV), torch.empty((16, N), device=DEV))
        x = torch.randn((M, K), generator=g).to(torch.bfloat16)
        out = torch.full((M + 1, N), 7.0, device=DEV)
        ks.linear(x.to(DEV), w.to(DEV), out[:M])
        bound = K * 2.0**-24 * (x.double().abs() @ w.double().abs().t())
        assert bool(((out[:M].cpu().double() - x.double() @ w.double().t()).abs() <= bound).all()) and bool((out[M] == 7.0).all())
        # the same rows dealt out to two of three groups, added to what is there
        first = (M + 1) // 2
        offsets = torch.tensor([0, first, first, M], dtype=torch.int32, device=DEV)
        h = torch.zeros((M, N), device=DEV)
        ks.grouped_linear_accumulate(x.to(DEV), w3, torch.arange(M, dtype=torch.int32, device=DEV), offsets, h)
        ref = torch.cat([x[:first].double() @ w.double().t(), x[first:].double() @ w.roll(2, 0).double().t()])
        bound = K * 2.0**-24 * torch.cat([x[:first].double().abs() @ w.double().abs().t(), x[first:].double().abs() @ w.roll(2, 0).double().abs().t()])
        assert bool(((h.cpu().double() - ref).abs() <= bound).all())
        calls += 3
    assert ks.launches_by_library["gemm_stream"] == before + calls and ks.errors() == {}
