"""The kernel that brings a decode step's integer inputs from pinned memory: whole numbers, so the same words; what it does not take is
left to the copy."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kernels():
    from spite_b200.kernels.cuda import CudaKernels
    return CudaKernels(torch.bfloat16, "cuda:0")


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 1024, 1025, 4099, 32768])
def test_words_arrive(kernels, n):
    host = torch.randint(-2**31, 2**31 - 1, (n,), dtype=torch.int32).pin_memory()
    out = torch.full((n + 4,), 7, dtype=torch.int32, device="cuda")
    assert kernels.upload_words(host, out[:n])
    assert torch.equal(out[:n].cpu(), host) and out[n:].eq(7).all()


def test_what_the_copy_keeps(kernels):
    out = torch.empty(32772, dtype=torch.int32, device="cuda")
    assert not kernels.upload_words(torch.zeros(8, dtype=torch.int32), out[:8])                          # pageable memory
    pinned = torch.zeros(32772, dtype=torch.int32).pin_memory()
    assert not kernels.upload_words(pinned[1:9], out[:8]) and not kernels.upload_words(pinned[:8], out[1:9])     # off a 16-byte boundary
    assert not kernels.upload_words(pinned[:32769], out[:32769]) and not kernels.upload_words(pinned[:8], out[:9])
