"""Decode products of 17 to 32 rows (tokens that arrive as boxes, up to four k slices a stage) against float64."""
import pytest
import torch

DEV = "cuda:0"


def data(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16)
    w = torch.randn((N, K), generator=g).to(torch.bfloat16)
    return x, w


@pytest.mark.gpu
@pytest.mark.parametrize("force", [(1, 2), (2, 4), (4, 1), (4, 2), (4, 3), None], ids=str)
@pytest.mark.parametrize("M,N,K", [(17, 40, 512), (24, 200, 1024), (32, 129, 2048), (31, 2048, 2048), (20, 96, 256)])
def test_products_of_17_to_32_rows(force, M, N, K):
    from spite_b200.kernels.cuda import CudaKernels
    ks = CudaKernels(torch.bfloat16, DEV)
    ks.stream_force = force
    x, w = data(M, N, K)
    before = ks.launches_by_library["gemm_stream"]
    # rows of a larger buffer: what lies behind the tokens must not be read as a token
    rows = torch.full((M + 40, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    rows[:M] = x.to(DEV)
    out = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=DEV)
    ks.linear(rows[:M], w.to(DEV), out[:M])
    again = torch.empty((M, N), dtype=torch.float32, device=DEV)
    ks.linear(x.to(DEV), w.to(DEV), again)
    ref = x.double() @ w.double().t()
    # a float32 sum of K products of magnitude |x||w|: each of its at most K roundings is below 2^-24 of the sum of magnitudes
    bound = K * 2.0**-24 * (x.double().abs() @ w.double().abs().t())
    assert bool(((out[:M].cpu().double() - ref).abs() <= bound).all())
    assert bool((out[M] == 7.0).all()) and torch.equal(again, out[:M])
    F = N // 2
    a = torch.empty((M, F), dtype=torch.bfloat16, device=DEV)
    ks.linear_swiglu(x.to(DEV), w[:2 * F].contiguous().to(DEV), a)
    gate, up = ref[:, :F], ref[:, F:2 * F]
    want = gate / (1 + torch.exp(-gate)) * up
    # bfloat16 rounding of the result (2^-8) and the two sums' bounds through silu (slope below 1.1) and the product
    tol = 2.0**-8 * want.abs() + 1.1 * bound[:, :F] * up.abs() + bound[:, F:2 * F] * gate.abs() + 1e-5 * want.abs() + 1e-6
    assert bool(((a.cpu().double() - want).abs() <= tol).all())
    assert ks.launches_by_library["gemm_stream"] == before + 3 and ks.errors() == {}


def test_stream_handles_without_the_undocumented_name(monkeypatch):
    from types import SimpleNamespace
    from spite_b200.kernels.cuda import CudaKernels
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 100 + device, raising=False)
    assert CudaKernels._raw_stream() == 103
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=77))
    assert CudaKernels._raw_stream() == 77
