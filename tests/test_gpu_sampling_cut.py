"""The cuts of top-k and top-p on the device: rows spread over a cluster's shared memory, at the sizes where a thread's share is odd, even
(padded) or nothing, and over the logits that the search by bins, its proof and its fall-back meet."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rows_of(kind, R, V, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn((R, V), generator=g)
    if kind == "even":
        return x * 2.5
    if kind == "narrow":                                     # thousands of logits in every bin: the bins are made narrower
        return x * 0.02
    if kind == "wide":                                       # the cut lies further below the maximum than the first bins reach
        return x * 0.5 + torch.where(torch.arange(V) == V // 2, 18.0, 0.0)
    if kind == "packed":                                     # ... three times, far below the maximum
        return torch.where(torch.arange(V) == V // 2, 5.0, 2.0**-10 + 2.0**-15 * torch.rand((R, V), generator=g))
    if kind == "ties":                                       # hundreds of equal logits at the cut
        return (x * 2).round() / 2
    if kind == "equal":                                      # nothing but equal logits: the search bit by bit
        return torch.full((R, V), 0.75)
    if kind == "zeros":                                      # zeros of both signs around the cut
        return torch.where(x.abs() < 0.7, torch.zeros(()), x) * torch.where(torch.rand((R, V), generator=g) < 0.5, 1.0, -1.0)
    if kind == "sorted":                                     # all candidates in one block
        return (x * 2.5).sort(1, descending=True).values
    assert kind == "masked"                                  # most of the row is gone
    return torch.where(torch.rand((R, V), generator=g) < 0.97, torch.tensor(-float("inf")), x * 2.5)


@pytest.mark.parametrize("V", [7, 33, 4096, 50257, 202048, 262144])
@pytest.mark.parametrize("kind", ["even", "narrow", "wide", "packed", "ties", "equal", "zeros", "sorted", "masked"])
@pytest.mark.parametrize("with_min_p", [False, True], ids=["", "min_p"])
def test_drawn_tokens_lie_behind_the_cuts(kind, V, with_min_p):
    """The token must be one that top-k and top-p keep, and the one whose part of the kept mass, in index order, holds u times that mass;
    both against 64 bits.  A float32 sum here goes through at most 49 + 5 + 5 + 8 additions in a row and expf errs by 2 units, so a
    mass is off by at most 70 * 2^-24 = 4.2e-6 of the whole; with the cut and the draw both off, 2e-5 is allowed."""
    from plain_llama4 import lcg_next
    from spite_b200.kernels.cuda import CudaKernels
    ks = CudaKernels(torch.float32, DEV)
    R = 16
    logits = rows_of(kind, R, V, V + len(kind))
    if V > 8:
        logits[:, 3] = 1.0                                   # (a masked row keeps at least one)
    else:
        logits[:, 0] = 1.0
    temperature = torch.tensor([0.6, 1.0, 1.7, 0.9] * 4)
    top_k = torch.tensor([0, 0, 0, 40, 0, 1, V // 3 + 1, 1000, 0, 0, 20000, 2, 0, V - 1, 0, 5], dtype=torch.int32)
    top_p = torch.tensor([0.9, 0.95, 0.5, 0.9, 0.999, 1.0, 0.8, 1.0, 0.3, 0.01, 0.95, 0.6, 0.99999, 0.7, 1.0, 0.95])
    min_p = torch.tensor([0.0, 0.05, 0.01, 1.0, 1e-4, 0.3, 0.02, 1.0, 0.001, 0.1, 1e-6, 0.5, 0.003, 0.2, 1.0, 0.0]) if with_min_p else torch.zeros(R)
    state = torch.arange(R, dtype=torch.int64) * 987654321987 + 5
    dev_state = state.to(DEV)
    got = ks.sample(logits.to(DEV), temperature=temperature.to(DEV), top_k=top_k.to(DEV), top_p=top_p.to(DEV), rng_state=dev_state,
                    **({"min_p": min_p.to(DEV)} if with_min_p else {})).cpu()
    slack = 2e-5
    for r in range(R):
        new, u = lcg_next(int(state[r]))
        assert int(dev_state[r]) & ((1 << 64) - 1) == new
        x32 = (logits[r] / temperature[r]).numpy()           # the division is the pipeline's, in float32
        if min_p[r] > 0:                                     # ... and so is this comparison
            x32 = np.where(x32 < x32.max() + np.log(min_p[r].numpy()), np.float32(-np.inf), x32)
        x, k = x32.astype(np.float64), int(top_k[r])
        # downwards; the device takes 0 before -0, in both cuts, and of equal logits the lower index first
        order = np.lexsort((np.arange(V), np.signbit(x32), -x))
        if 0 < k < V:
            kth = order[k - 1]
            gone = (x < x[kth]) | ((x == x[kth]) & np.signbit(x32) & ~np.signbit(x32[kth]))
            x = np.where(gone, -np.inf, x)
        mass = np.exp(x - x.max())
        token = int(got[r])
        assert mass[token] > 0
        # what lies within the allowance of the wanted mass may be kept or not: the draw must fit one of the kept sets between
        around = [float(np.float32(top_p[r])) * mass.sum() + s * slack * mass.sum() for s in (-1, 0, 1)] if float(top_p[r]) < 1 else [np.inf]
        before = np.concatenate([[0.0], np.cumsum(mass[order])[:-1]])
        place = np.nonzero(order == token)[0][0]
        assert before[place] < around[-1], (r, "behind the cut of top-p")
        fits = []
        for want in around:
            kept = np.zeros(V, bool)
            kept[order[(before < want) | (np.arange(V) == place)]] = True
            cum = np.cumsum(np.where(kept, mass, 0.0))
            target = u * cum[-1]
            fits.append(cum[token] - mass[token] - slack * mass.sum() <= target <= cum[token] + slack * mass.sum())
        assert any(fits), (r, token)


@pytest.mark.parametrize("V", [33, 4096, 50257, 202048])
def test_rows_with_numbers_that_are_not_finite(V):
    """A row with NaN or +inf, or with nothing but -inf, gives some token of the vocabulary, the same each time, advances its state and leaves the
    other rows alone; the argmax finds +inf (of several the last), and what is masked out is not drawn where anything else is left."""
    from plain_llama4 import lcg_next
    from spite_b200.kernels.cuda import CudaKernels
    ks, g, nan, inf = CudaKernels(torch.float32, DEV), torch.Generator().manual_seed(V), float("nan"), float("inf")
    some = torch.randperm(V, generator=g)[:5]
    odd = [lambda x: x.index_fill_(0, some[:1], nan), lambda x: x.index_fill_(0, some, inf), lambda x: x.fill_(nan), lambda x: x.fill_(-inf),
           lambda x: x.fill_(-inf).index_fill_(0, some[:2], nan), lambda x: x.index_fill_(0, some[:1], nan).index_fill_(0, some[1:2], inf),
           lambda x: x.fill_(-inf).index_fill_(0, some[:1], 2.0), lambda x: x.fill_(inf), lambda x: x.fill_(-inf).index_fill_(0, some, inf)]
    for T, k, p, m in [(1.0, 0, 1.0, 0.0), (0.7, 0, 0.9, 0.0), (1.0, 7, 1.0, 0.0), (1.3, 7, 0.8, 0.0), (1.0, 7, 0.8, 0.05), (1.0, 0, 0.9, 1.0), (1.0, 0, 1.0, 0.1),
                       (0.0, 0, 1.0, 0.0), (0.0, 7, 0.9, 0.1), (0.0, 0, 0.5, 1.0)]:
        plain = torch.randn((2 * len(odd), V), generator=g) * 2
        logits = plain.clone()
        for i, change in enumerate(odd):
            change(logits[2 * i])
        R = logits.shape[0]
        results = []
        for given in (logits, logits, plain):
            state = torch.arange(R, device=DEV) * 1234567 + 3
            one = lambda v, t=torch.float32: torch.full((R,), v, dtype=t, device=DEV)
            token = ks.sample(given.to(DEV), temperature=one(T), top_k=one(k, torch.int32), top_p=one(p), min_p=one(m), rng_state=state)
            results.append((token.tolist(), [s & (1 << 64) - 1 for s in state.tolist()]))
        tokens, states = results[0]
        assert results[1] == results[0] and tokens[1::2] == results[2][0][1::2]
        assert states == [lcg_next(r * 1234567 + 3)[0] if T > 0 else r * 1234567 + 3 for r in range(R)]
        assert all(0 <= t < V for t in tokens)
        assert tokens[12] == int(some[0])                    # the only logit that is not masked
        if T <= 0:
            assert tokens[2] == tokens[16] == int(some.max()) and tokens[14] == V - 1
