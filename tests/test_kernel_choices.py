"""How the weight-streaming kernel's work is cut (ring, k slices inside a block, k splits across blocks): the kernel set's own choice on the host,
at shapes it was measured on and at its borders.  The kernel itself with every cut:
test_gpu_kernels.py::test_streaming_products_with_k_slices_and_k_splits."""
import pytest

from spite_b200.kernels.cuda import CudaKernels, stream_cut

DEEP, OTHER = CudaKernels.stream_rings(148)


def chooser(**changed):
    ks = object.__new__(CudaKernels)                          # the choice alone: no device
    ks.stream_shape, ks.stream_force = ks.stream_rings(148), None
    for name, value in changed.items():
        assert hasattr(ks, name)
        setattr(ks, name, value)
    return ks


def plan(M, N, K, swiglu=False, experts=0, ks=None):
    return (ks or chooser())._stream_plan(M, N, K, experts or 1, swiglu, M, experts > 0, False)


def cut(*args, **kw):
    return plan(*args, **kw)[3:5]


# rows, N, K, SwiGLU, experts: the cuts within 5 % of the fastest of all, each measured behind a norm in a graph over several layers' weights
MEASURED = [
    ((1, 7168, 5120, False, 0), {(4, 1), (1, 4), (1, 3), (2, 2)}), ((8, 7168, 5120, False, 0), {(4, 1), (1, 4)}),
    ((1, 5120, 5120, False, 0), {(1, 6), (1, 7), (2, 3), (1, 3)}), ((8, 5120, 5120, False, 0), {(1, 4), (1, 3), (2, 3)}),
    ((8, 5120, 8192, False, 0), {(1, 4), (2, 3), (1, 3)}), ((8, 4096, 4096, False, 0), {(8, 1), (4, 2), (1, 4)}),
    ((4, 8192, 2048, False, 0), {(4, 1), (1, 4)}), ((16, 8192, 2048, False, 0), {(4, 1)}),
    ((1, 2048, 2048, False, 0), {(1, 8), (8, 1), (1, 7), (2, 4), (2, 8), (4, 4)}), ((4, 2048, 2048, False, 0), {(2, 4), (4, 4), (2, 8), (4, 2), (8, 1)}),
    ((24, 2048, 2048, False, 0), {(4, 4), (4, 3)}), ((24, 5120, 16384, False, 0), {(2, 3)}), ((24, 8192, 2048, True, 0), {(2, 1)}),
    ((1, 8192, 5120, True, 0), {(2, 1), (1, 2)}), ((8, 8192, 5120, True, 0), {(2, 1), (1, 2)}), ((3, 4864, 8192, True, 0), {(1, 3)}),
    ((8, 12544, 12288, False, 0), {(2, 1), (1, 2), (1, 3)}),
    ((8, 1024, 2048, True, 32), {(2, 1)}), ((8, 2048, 1024, False, 32), {(2, 1)}), ((16, 2048, 2048, False, 16), {(2, 1), (1, 2), (4, 1)}),
    ((3, 1024, 2048, True, 16), {(4, 1), (1, 4), (1, 3), (2, 3)}), ((1, 8192, 5120, True, 16), {(2, 1), (1, 2)}),
    ((8, 8192, 5120, True, 16), {(2, 1), (1, 1), (4, 1), (1, 2), (2, 2)}), ((8, 5120, 8192, False, 16), {(4, 1), (1, 4), (2, 3), (1, 3), (1, 1)})]     # (the last 6 %)


@pytest.mark.parametrize("shape,fast", MEASURED, ids=lambda v: "x".join(str(int(x)) for x in v) if isinstance(v, tuple) else "")
def test_the_measured_shapes_get_a_cut_among_the_fastest(shape, fast):
    assert cut(*shape) in fast


def test_the_ring():
    """One-group products and few rows run in the deeper ring, experts' products of four to eight rows while their weights are few."""
    ring = lambda *a, **kw: plan(*a, **kw)[:2]
    assert all(ring(M, 7168, 5120) == DEEP for M in (1, 8, 16, 24, 32))
    assert all(ring(M, 8192, 5120, True, 16) == (DEEP if M <= 3 else OTHER) for M in range(1, 17))
    assert all(ring(M, 1024, 2048, True, 32) == (DEEP if M <= 8 else OTHER) for M in range(1, 17))          # 60 MB at eight rows
    likely = 16 * (1 - (15 / 16) ** 8)                        # experts that eight rows reach of 16
    at_line = int(CudaKernels.stream_deep_bytes / (likely * 4096 * 2))
    assert ring(8, at_line, 4096, False, 16) == DEEP and ring(8, at_line + 1, 4096, False, 16) == OTHER


@pytest.mark.parametrize("M", [1, 2, 3, 4, 6, 8, 9, 13, 16, 17, 24, 32])
@pytest.mark.parametrize("N,K,swiglu", [(40, 64, False), (200, 320, False), (104, 1024, True), (5120, 8192, False), (2048, 2048, False),
                                        (8192, 5120, True), (129, 4096, False), (16, 64, True), (1024, 16384, False), (202048, 5120, False)])
@pytest.mark.parametrize("experts", [0, 2, 8, 128])
def test_every_cut_is_one_the_kernel_takes(M, N, K, swiglu, experts):
    if experts and M > 16:
        return                                                 # grouped products of more rows go elsewhere
    smem, blocks, nt, slices, splits, cluster = plan(M, N, K, swiglu, experts)
    assert (smem, blocks) in (DEEP, OTHER) and nt == (8 if M <= 8 else 16 if M <= 16 else 32)
    assert slices in (1, 2, 4, 8) and K % (64 * slices) == 0          # a stage is `slices` k blocks of 64
    assert not (swiglu and slices == 8) and not (nt == 32 and slices == 8)     # tiles that are not built
    assert 1 <= splits <= min(16, K // (64 * slices))                  # no split without a stage
    assert not cluster or slices == 1 and 2 <= splits <= 4 and nt < 32
    fixed = 24 * 8 + 16 + 4 * (1 if nt == 32 else 1024) + (8 - 8 // slices) * 64 * nt * (slices > 1) + 1024
    assert (smem - fixed) // (16384 + max(1024, slices * nt * 128)) >= 2       # a ring of at least two stages fits


def test_splits_that_can_be_a_cluster():
    """The cost of a cluster is asked only of so many splits as a cluster may have, without slices, whose blocks are all resident at once."""
    kw = dict(CudaKernels.stream_costs, split_item_cost=1000.0, cluster_cost=0.0, slice_each=1000.0, lone_rate=1.25, lone_rate_slices=1.25)
    one = lambda N, groups=1, most=1, clusters=4: stream_cut(N, 5120, groups, most, False, 296, DEEP[0], 8, 8, clusters, **kw)
    assert one(7168) == (1, 4) and one(7168, clusters=3) == (1, 3) and one(7168, clusters=0) == (1, 1)
    assert one(128 * 75) == (1, 3)                                     # 75 tiles in fours are 300 blocks for 296 places
    assert one(128 * 37, 1.9, 2) == (1, 4) and one(128 * 38, 1.9, 2) == (1, 3)        # ... of all groups that there may be
    # up to four splits in the deeper ring, two in the other, none beyond stream_cluster_max_rows rows
    assert plan(1, 5120, 2048, True)[3:] == (1, 3, True) and plan(1, 5120, 2048, True, ks=chooser(stream_cluster_max_rows=0))[3:] == (1, 3, False)
    clusters = {(M, *plan(M, N, 5120, sw, E)[4:]) for M in (1, 8, 16) for N in range(512, 16384, 128) for sw in (False, True) for E in (0, 16)}
    assert all(splits <= 4 for M, splits, cluster in clusters if cluster) and any(cluster and splits == 4 for _, splits, cluster in clusters)
    assert not any(cluster and splits > 2 for N in range(512, 8192, 128) for *_, splits, cluster in [plan(16, N, 5120, False, 16)])


def test_a_choice_made_for_every_call():
    assert cut(8, 5120, 5120, ks=chooser(stream_force=(4, 2))) == (4, 2)
