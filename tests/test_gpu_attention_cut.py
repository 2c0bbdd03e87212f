"""Prompt-portion attention on the tcgen05 kernel with its work cut along the keys: whole items and cut ones against float64, in every form the
kernel has.  The tolerance is the one of the kernel's other tests (weights and outputs in bfloat16)."""
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


def run(ks, monkeypatch, cut, *args, **kw):
    monkeypatch.setattr(cuda_kernels, "attention_cut_pays", lambda *a: cut)
    q, out, batch, cache = args
    out.fill_(float("nan"))
    ks.attention_scratch_bytes = 0
    ks.paged_attention(q, out, batch, cache, **kw)
    torch.cuda.synchronize()
    assert not ks.errors()
    return out.clone(), ks.attention_scratch_bytes


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
    cut, scratch = run(ks, monkeypatch, True, *args, **kw)
    assert scratch >= ks.sm_count * 4 * (hd + 2) * 128 * 4
    again, _ = run(ks, monkeypatch, True, *args, **kw)                 # the parts are added in one order
    assert torch.equal(cut, again)
    whole, _ = run(ks, monkeypatch, False, *args, **kw)
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
    cut, scratch = run(ks, monkeypatch, True, *args, **kw)
    whole, none = run(ks, monkeypatch, False, *args, **kw)
    assert scratch >= ks.sm_count * 4 * (hd + 2) * 128 * 4 > none or len(specs) > 1
    close(cut, whole, TOL[torch.bfloat16], form)
