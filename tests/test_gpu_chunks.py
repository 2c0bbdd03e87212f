"""Recurrences in chunks of 32 tokens on the tensor cores (GPU), against float64 walked token by token: chunk edges, remainders,
segments short enough for the walk token by token beside long ones, sizes that fill no tile, states carried from step to step, gates
that erase everything, numbers that are not finite.

The tolerance: float32 walked token by token is within 2e-5 of float64 in these cases (the other recurrence tests), and a split
operand holds 2^-23 of a number, so the chunks get the same."""
import ctypes as C

import pytest
import torch

from test_gpu_gapevik import DEV, kernels, step_batch

pytestmark = pytest.mark.gpu
TOL = 2e-5


def near(got, want, what, tol=TOL):
    want = want.to(got.device)
    assert torch.isfinite(got).all(), what
    err = (got.double() - want).abs().max() / max(float(want.abs().max()), 1e-30)
    assert err <= tol, f"{what}: {float(err):.2e}"


# ---------------------------------------------------------------------------- the gated delta rule
def delta_reference(x, cols, heads, kvh, dim, vdim, a_log, dt, q_scale, S):
    """One segment token by token in float64; S [heads, dim, vdim] -> (outputs [T, heads, vdim], S)."""
    x, T, rep = x.double(), x.shape[0], heads // kvh
    q = x[:, cols[0]:cols[0] + kvh * dim].view(T, kvh, dim).repeat_interleave(rep, 1)
    k = x[:, cols[1]:cols[1] + kvh * dim].view(T, kvh, dim).repeat_interleave(rep, 1)
    v = x[:, cols[2]:cols[2] + heads * vdim].view(T, heads, vdim)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * q_scale
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(x[:, cols[3]:cols[3] + heads])
    g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(x[:, cols[4]:cols[4] + heads] + dt.double()))
    out = torch.zeros_like(v)
    for t in range(T):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out, S


# (heads, kv heads, dim, vdim, segments as token counts of two steps)
DELTA = [
    (2, 1, 128, 128, [(64, 1), (33, 31), (1, 95)]),
    (3, 3, 20, 12, [(32, 17), (15, 16), (129, 2)]),
    (4, 2, 72, 140, [(31, 65), (16, 1)]),
    (1, 1, 64, 5, [(250, 97)]),
    (48, 12, 128, 64, [(40, 33), (70, 1), (18, 20)]),
]


@pytest.mark.parametrize("case", range(len(DELTA)))
@pytest.mark.parametrize("gates", ["mild", "harsh"])
def test_delta_rule_in_chunks(case, gates):
    heads, kvh, dim, vdim, segs = DELTA[case]
    ks = kernels(torch.bfloat16)
    ks.chunk_min_tokens = 16
    g = torch.Generator().manual_seed(11 + case)
    slots = torch.randperm(len(segs) + 2, generator=g)[:len(segs)].tolist()
    state = torch.randn((len(segs) + 2, 8 + heads * dim * vdim + 3), generator=g).to(DEV)
    state[slots] = 0.0
    a_log = (torch.randn(heads, generator=g) * 0.7 - 1.0 if gates == "mild" else torch.randn(heads, generator=g) * 4.0).to(DEV)
    dt = torch.randn(heads, generator=g).to(DEV)
    cols = (3, 3 + kvh * dim, 3 + 2 * kvh * dim, 5 + 2 * kvh * dim + heads * vdim, 5 + 2 * kvh * dim + heads * vdim + heads)
    carried = [torch.zeros((heads, dim, vdim), dtype=torch.float64, device=DEV) for _ in segs]
    for step in range(2):
        counts = [s[step] for s in segs]
        batch, M = step_batch(counts, slots, step == 0)
        x = torch.randn((M, cols[4] + heads + 2), generator=g).to(DEV)
        x[:, cols[3]:] *= 3.0 if gates == "mild" else 10.0
        x[:, cols[2]:cols[3]] *= 1e-3 if case % 2 else 1e3
        out = torch.empty((M, heads * vdim), dtype=torch.float32, device=DEV)
        ks.delta_scan(x, out, batch, state, heads=heads, kv_heads=kvh, dim=dim, vdim=vdim, columns=cols, a_log=a_log, dt_bias=dt,
                      q_scale=dim ** -0.5, state_offset=8, chunked=True)
        off = 0
        for s, n in enumerate(counts):
            ref, carried[s] = delta_reference(x[off:off + n], cols, heads, kvh, dim, vdim, a_log, dt, dim ** -0.5, carried[s])
            near(out[off:off + n].view(n, heads, vdim), ref, f"step {step}, segment {s}")
            near(state[slots[s], 8:8 + heads * dim * vdim].view(heads, dim, vdim), carried[s], f"step {step}, state of segment {s}")
            off += n


@pytest.mark.parametrize("where", ["value", "key", "state"])
def test_delta_rule_with_an_infinity_is_walked_token_by_token(where):
    """What stands before a number that is not finite stays as it is, other heads and segments too; the walk in chunks gives what
    the walk token by token gives."""
    heads, dim, vdim, counts = 2, 64, 32, [70, 40]
    ks = kernels(torch.bfloat16)
    g = torch.Generator().manual_seed(5)
    cols = (0, dim * heads, 2 * dim * heads, 2 * dim * heads + heads * vdim, 2 * dim * heads + heads * vdim + heads)
    batch, M = step_batch(counts, [0, 1], True)
    x = torch.randn((M, cols[4] + heads), generator=g).to(DEV)
    if where != "state":
        x[50, (cols[2] if where == "value" else cols[1]) + 3] = float("inf")              # head 0, first segment
    outs, states = [], []
    for chunked in (True, False):
        state = torch.zeros((2, heads * dim * vdim), device=DEV)
        if where == "state":
            state[0, 3 * vdim + 20] = float("inf")
        out = torch.empty((M, heads * vdim), device=DEV)
        ks.delta_scan(x, out, batch, state, heads=heads, kv_heads=heads, dim=dim, vdim=vdim, columns=cols, a_log=torch.zeros(heads, device=DEV),
                      dt_bias=torch.zeros(heads, device=DEV), q_scale=1.0, chunked=chunked)
        outs.append(out)
        states.append(state)
    part = slice(0, vdim) if where != "state" else slice(16, vdim)        # (the columns that the infinity reaches)
    torch.testing.assert_close(outs[0][:70, part], outs[1][:70, part], rtol=TOL, atol=0, equal_nan=True)
    assert not torch.isfinite(outs[0][:70, part]).all()
    torch.testing.assert_close(states[0][0], states[1][0], rtol=1e-3, atol=1e-4, equal_nan=True)
    if where != "state":
        near(outs[0][:50], outs[1][:50].double(), "before the infinity")
    near(outs[0][:, vdim:], outs[1][:, vdim:].double(), "the other head")
    near(states[0][1], states[1][1].double(), "the other segment's state")


def test_delta_entry_points_refuse_malformed_calls():
    from spite_b200.kernels import build
    from spite_b200.kernels.cuda import DeltaParams
    lib = build.load("delta")
    lib.spite_delta_chunk_bytes.restype = C.c_longlong
    assert lib.spite_delta_chunk_bytes(129, 8, 1, 1, 10, 1, 1) == -2 and lib.spite_delta_chunk_bytes(0, 8, 1, 1, 10, 1, 1) == -1
    t = torch.zeros(1 << 16, device=DEV)
    a = dict.fromkeys(("x", "a_log", "dt_bias", "out", "state", "cu_seqlens", "slots", "gates"), t.data_ptr())
    a.update(stride=200, q_col=0, k_col=16, v_col=32, b_col=48, a_col=49, slot_stride=256, n_segments=1, heads=1, kv_heads=1, dim=16, vdim=16,
             q_scale=1.0, unit_eps=1e-6, n_tokens=4)
    call = lambda scratch=t.data_ptr(), chunks=1, least=1, **k: lib.spite_delta_scan_chunked(C.byref(DeltaParams(**dict(a, **k))), C.c_void_p(scratch),
                                                                                             chunks, least, None)
    assert call(scratch=None) == -1 and call(scratch=t.data_ptr() + 4) == -1 and call(chunks=0) == -1 and call(least=0) == -1
    assert call(dim=160, stride=2000, k_col=160, v_col=320, slot_stride=1 << 14) == -2 and call(heads=0) == -1
    assert call(n_segments=0) == 0
    torch.cuda.synchronize()
    assert not t.any()
