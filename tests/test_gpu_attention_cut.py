"""Prompt-portion attention on the tcgen05 kernel with its work cut along the keys: whole items and cut ones against float64, in every form the
kernel has.  The tolerance is the one of the kernel's other tests (weights and outputs in bfloat16)."""
import ctypes as C
import math

import pytest
import torch

from spite_b200.cache import LayerCache, Window
from spite_b200.kernels import cuda as cuda_kernels
from test_gpu_kernels import TOL, close, dense_attention_reference, fill_cache, make_batch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# query heads, kv heads, head size, page, window, (first position, tokens) of every request
CASES = [
    (10, 2, 128, 64, ("full", 0), [(5000, 60)]),                       # few long items: an item has a dozen parts, the second row tile 10 tokens
    (10, 2, 128, 64, ("full", 0), [(20000, 25)]),                      # no token in the second row tile
    (40, 8, 128, 64, ("chunk", 8192), [(3000, 700)]),                  # more items than blocks
    (16, 1, 64, 64, ("full", 0), [(0, 1500)]),                         # items of 1 to 24 tiles: some shorter than a part may be
    (4, 4, 64, 128, ("sliding", 300), [(900, 700), (0, 140)]),         # windows: parts without a key for one of the row tiles
    (6, 2, 128, 64, ("chunk", 512), [(400, 900), (3, 5), (5000, 64), (77, 1)]),     # beside segments that other kernels serve
    (3, 3, 128, 64, ("full", 0), [(1000, 128)]),
]


def run(ks, monkeypatch, cut, *args, takes=True, **kw):
    """One call with the choice made: a cut call launches a second kernel that adds the parts up (unless the cut form does not take the call)."""
    monkeypatch.setattr(cuda_kernels, "attention_cut_pays", lambda *a: cut)
    q, out, batch, cache = args
    out.fill_(float("nan"))
    before = ks.launches_by_library["attention_tc"]
    ks.paged_attention(q, out, batch, cache, **kw)
    torch.cuda.synchronize()
    assert not ks.errors() and ks.launches_by_library["attention_tc"] == before + 1 + (cut and takes)
    return out.clone()


@pytest.mark.parametrize("case", range(len(CASES)))
def test_cut_along_the_keys(case, monkeypatch):
    nq, nkv, hd, P, window, specs = CASES[case]
    ks, win = cuda_kernels.CudaKernels(torch.bfloat16, DEV), Window(*window)
    n_pages = sum(-(-(s + n) // P) for s, n in specs) + 5
    batch, tables = make_batch(specs, P, n_pages, 40 + case, DEV)
    M, g = batch.n_tokens, torch.Generator().manual_seed(41 + case)
    k_all = [torch.randn((s + n, nkv, hd), generator=g).to(torch.bfloat16) for s, n in specs]
    v_all = [torch.randn((s + n, nkv, hd), generator=g).to(torch.bfloat16) for s, n in specs]
    q = torch.randn((M, nq, hd), generator=g)
    q[3] = k_all[0][win.lowest_visible(specs[0][0] + 3) + 1, 0].float() * (14.0 / math.sqrt(hd))    # one far key carries a row: one part decides
    q = q.to(torch.bfloat16)
    kv = torch.zeros((2, n_pages, nkv, P, hd), dtype=torch.bfloat16)
    fill_cache(kv, tables, [(s + n, 0) for s, n in specs], k_all, v_all, P)
    out, scale = torch.empty((M, nq * hd), dtype=torch.bfloat16, device=DEV), 1.0 / math.sqrt(hd)
    args = (q.reshape(M, nq * hd).to(DEV), out, batch, LayerCache(0, kv.to(DEV), None, P, False))
    kw = dict(num_heads=nq, window=win, softmax_scale=scale)
    cut = run(ks, monkeypatch, True, *args, **kw)
    assert len(specs) > 1 or ks.attention_scratch_bytes >= ks.sm_count * 4 * (hd + 2) * 128 * 4     # (other kernels set their own behind it)
    assert torch.equal(cut, run(ks, monkeypatch, True, *args, **kw))         # the parts are added in one order
    whole = run(ks, monkeypatch, False, *args, **kw)
    ref = dense_attention_reference(q, k_all, v_all, specs, nq, nkv, win, scale)
    close(whole.view(M, nq, hd), ref, TOL[torch.bfloat16], "whole items")
    close(cut.view(M, nq, hd), ref, TOL[torch.bfloat16], "cut items")


@pytest.mark.parametrize("form", ["sinks", "slopes", "gates by head", "cap", "distances", "keys alone"])
@pytest.mark.parametrize("case", [0, 4, 5])
def test_every_form_cut_as_whole(case, form, monkeypatch):
    """What joins once per row (sinks, gates) or per score, and the forms that are compiled apart, against the uncut kernel."""
    from spite_b200.kernels.api import DistanceBias
    nq, nkv, hd, P, window, specs = CASES[case]
    ks, win = cuda_kernels.CudaKernels(torch.bfloat16, DEV), Window(*window)
    n_pages = sum(-(-(s + n) // P) for s, n in specs) + 5
    batch, _ = make_batch(specs, P, n_pages, 60 + case, DEV)
    M, g = batch.n_tokens, torch.Generator(device=DEV).manual_seed(61 + case)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    kv, q = rnd(2, n_pages, nkv, P, hd).to(torch.bfloat16), rnd(M, nq * hd).to(torch.bfloat16)
    kw, factors = {}, None
    if form == "sinks":
        kw = dict(head_sinks=rnd(nq) * 4)
    elif form == "slopes":
        kw = dict(head_slopes=rnd(nq).abs() * 0.01)
    elif form == "gates by head":
        kw = dict(head_gates=rnd(M, nq).sigmoid(), out_by_head=True)
    elif form == "cap":
        kw = dict(score_softcap=2.0)
    elif form == "distances":
        kw = dict(distance_bias=DistanceBias.from_rows(rnd(20, nq), [min(n // 40, 19) for n in range(200)]), score_softcap=5.0)
    else:
        kv, factors = kv[:1].contiguous(), rnd(n_pages, nkv, P).abs() + 0.5
    out = torch.empty((M, nq * hd), dtype=torch.bfloat16, device=DEV)
    args = (q, out, batch, LayerCache(0, kv, None, P, False, factors))
    kw = dict(kw, num_heads=nq, window=win, softmax_scale=1.0 / math.sqrt(hd))
    cut = run(ks, monkeypatch, True, *args, **kw)
    whole = run(ks, monkeypatch, False, *args, **kw)
    close(cut, whole, TOL[torch.bfloat16], form)


def one_portion(ks, start, n, nq=40, nkv=8, hd=128, P=64):
    n_pages = -(-(start + n) // P) + 1
    batch, _ = make_batch([(start, n)], P, n_pages, 3, DEV)
    g = torch.Generator(device=DEV).manual_seed(start + n)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.empty((n, nq * hd), dtype=torch.bfloat16, device=DEV)
    return (rnd(n, nq * hd), out, batch, LayerCache(0, rnd(2, n_pages, nkv, P, hd), None, P, False)), \
        dict(num_heads=nq, window=Window("full", 0), softmax_scale=hd ** -0.5)


@pytest.mark.parametrize("start,n,cut", [(8092, 100, True), (7192, 1000, True), (0, 600, False), (500, 500, False)])
def test_the_rule_chooses(start, n, cut):
    """Without the choice made for it: the call asks the rule (whose answers are tested on the host) and follows it."""
    ks = cuda_kernels.CudaKernels(torch.bfloat16, DEV)
    args, kw = one_portion(ks, start, n)
    ks.paged_attention(*args, **kw)
    assert ks.launches_by_library["attention_tc"] == 1 + cut and (ks.attention_scratch_bytes > 0) == cut
    torch.cuda.synchronize()
    assert torch.isfinite(args[1]).all() and not ks.errors()


@pytest.mark.parametrize("n", [16384, 16385])
def test_more_pairs_of_row_tiles_than_are_cut(n, monkeypatch):
    """16 heads a kv head: 8 tokens a row tile, 1,024 pairs of them at 16,384 tokens; one more goes whole."""
    ks = cuda_kernels.CudaKernels(torch.bfloat16, DEV)
    args, kw = one_portion(ks, 0, n, nq=16, nkv=1, hd=64)
    takes = n <= 16384
    cut = run(ks, monkeypatch, True, *args, takes=takes, **kw)
    assert (ks.attention_scratch_bytes > 0) == takes
    whole = run(ks, monkeypatch, False, *args, **kw)
    close(cut, whole, TOL[torch.bfloat16], "cut")
    assert takes or torch.equal(cut, whole)


@pytest.mark.parametrize("cut", [False, True], ids=["whole", "cut"])
@pytest.mark.parametrize("kind", ["nan", "inf", "-inf"])
@pytest.mark.parametrize("place", [0, 6, 17, 30, 39, 48, 59, 63])
def test_a_score_that_is_no_number(place, kind, cut, monkeypatch):
    """A key whose score is NaN or +inf must show in every row that sees it, one whose score is -inf must weigh nothing, wherever in a tile of
    64 keys it stands: the weights of the places 6, 7, 16, 17, 26, 27 of every 32 are made on the multiply-add units, the others on the
    special-function units."""
    nq, nkv, hd, P, specs = 4, 2, 128, 64, [(900, 200)]
    ks, win, n_pages = cuda_kernels.CudaKernels(torch.bfloat16, DEV), Window("full", 0), 20
    batch, tables = make_batch(specs, P, n_pages, 7, DEV)
    M, g = batch.n_tokens, torch.Generator().manual_seed(place + len(kind))
    k, v = (torch.randn((1100, nkv, hd), generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn((M, nq, hd), generator=g).to(torch.bfloat16)
    q[:, :2] = -q[:, :2].abs() if kind == "-inf" else q[:, :2].abs()
    ref = dense_attention_reference(q[:, 2:], [k[:, 1:]], [v[:, 1:]], specs, 2, 1, win, hd ** -0.5)
    j = 256 + place
    others = torch.arange(1100) != j
    k[j, 0], v[j, 0] = float("nan") if kind == "nan" else 3e38, 1e38
    kv = torch.zeros((2, n_pages, nkv, P, hd), dtype=torch.bfloat16)
    fill_cache(kv, tables, [(1100, 0)], [k], [v], P)
    out = torch.empty((M, nq * hd), dtype=torch.bfloat16, device=DEV)
    got = run(ks, monkeypatch, cut, q.reshape(M, nq * hd).to(DEV), out, batch, LayerCache(0, kv.to(DEV), None, P, False), num_heads=nq, window=win,
                 softmax_scale=hd ** -0.5)
    got = got.view(M, nq, hd)
    close(got[:, 2:], ref, TOL[torch.bfloat16], "heads without that key")
    if kind != "-inf":
        assert bool(got[:, :2].isnan().all())
        return
    sc = torch.einsum("mhd,jd->hmj", q[:, :2].double(), k[others, 0].double()) * hd ** -0.5
    seen = torch.arange(1100)[others][None, :] <= 900 + torch.arange(M)[:, None]
    want = torch.softmax(sc.masked_fill(~seen, float("-inf")), -1) @ v[others, 0].double()
    close(got[:, :2], want.transpose(0, 1), TOL[torch.bfloat16], "without the key")


def test_powers_of_two():
    """The weights made on the multiply-add units.  The polynomial is within 7.5e-8 of 2^f and each of its five multiply-adds rounds by at most
    2^-24 of a result near 1, the first ones of a small part of it: 2.2e-7 in all over the range that weights have; below 2^-126 they may be
    off by half the smallest number, and what is no number stays none."""
    ks = cuda_kernels.CudaKernels(torch.bfloat16, DEV)
    x = torch.cat([torch.linspace(-126, 8, 1 << 20), torch.linspace(8, 127, 1 << 16)])
    special = torch.tensor([float("nan"), -float("inf"), -127.0, -1e30, -3e38, 0.0, 1.0, -126.0, float("inf"), float("nan"), 5.0, float("nan")])
    for given in (x, special):
        dev, y = given.to(DEV), torch.empty(given.numel(), device=DEV)
        assert ks._lib("attention_tc").spite_attention_exp2_pairs(C.c_void_p(dev.data_ptr()), C.c_void_p(y.data_ptr()), given.numel() // 2,
                                                                  ks._stream()) == 0
        y = y.cpu()
        if given is x:
            want = torch.exp2(x.double())
            assert float((y.double() / want - 1).abs().max()) <= 2.2e-7
        else:
            assert y.isnan().tolist() == [True] + 7 * [False] + [True, True, False, True]
            assert y[1:5].tolist() == [0.0] * 4 and bool(((y[5:8] / torch.tensor([1.0, 2.0, 2.0 ** -126]) - 1).abs() <= 2.2e-7).all())
