"""Recurrences in chunks of 32 tokens on the tensor cores (GPU), against float64 walked token by token: chunk edges, remainders,
segments short enough for the walk token by token beside long ones, sizes that fill no tile, states carried from step to step, gates
that erase everything, numbers that are not finite.

The tolerance: float32 walked token by token is within 2e-5 of float64 in these cases (the other recurrence tests), and a split
operand holds 2^-23 of a number down to 2^-28 of the largest in its sum, so the chunks get the same.  Numbers of very different size
have a test of their own, with errors relative to each column, token and key."""
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


# ---------------------------------------------------------------------------- the walks of scan.cu
def scan_reference(kind, q, k, v, w, extra, S):
    """One segment in float64, q, k [T, heads, dim], v [T, heads, vdim], S [heads, vdim, dim]."""
    out = torch.zeros_like(v)
    for t in range(q.shape[0]):
        kv = v[t][:, :, None] * k[t][:, None, :]
        if kind == "memory":
            out[t] = torch.einsum("hvk,hk->hv", S, q[t]) + (q[t] * extra * k[t]).sum(-1)[:, None] * v[t]
        S = w[t] * S + kv
        if kind != "memory":
            out[t] = torch.einsum("hvk,hk->hv", S, q[t])
    return out, S


# (heads, kv heads (state space), dim, vdim, segments as token counts of two steps)
SCANS = [
    (2, 1, 64, 64, [(64, 1), (33, 31), (1, 95)]),
    (3, 1, 20, 12, [(32, 17), (15, 16), (129, 2)]),
    (20, 1, 128, 70, [(31, 65), (16, 1)]),
    (2, 2, 100, 5, [(250, 97)]),
    (34, 2, 128, 64, [(40, 33), (70, 1), (18, 20)]),
]


@pytest.mark.parametrize("case", range(len(SCANS)))
@pytest.mark.parametrize("gates", ["mild", "harsh"])
@pytest.mark.parametrize("kind", ["state_space", "memory", "linear_attention"])
def test_scans_in_chunks(kind, gates, case):
    heads, kvh, dim, vdim, segs = SCANS[case]
    kvh = kvh if kind == "state_space" else heads
    ks = kernels(torch.bfloat16)
    ks.chunk_min_tokens = 16
    g = torch.Generator().manual_seed(50 + case)
    rnd = lambda *s: torch.randn(s, generator=g).to(DEV)
    size = heads * ks.scan_state_size(dim, vdim)
    dim4 = -(-dim // 4) * 4
    slots = torch.randperm(len(segs) + 2, generator=g)[:len(segs)].tolist()
    state = rnd(len(segs) + 2, 8 + size)
    state[slots] = 0.0
    harsh = 1.0 if gates == "mild" else 5.0
    carried = [torch.zeros((heads, vdim, dim), dtype=torch.float64, device=DEV) for _ in segs]
    a_log, dt, skip, w0, u = rnd(heads) * harsh - 1.0, rnd(heads), rnd(heads), rnd(heads * dim) * harsh - 2.0, rnd(heads * dim)
    a2, a2_bias = rnd(6, heads * dim), rnd(heads * dim) * harsh
    for step in range(2):
        counts = [s[step] for s in segs]
        batch, M = step_batch(counts, slots, step == 0)
        q, k, v = rnd(M, kvh * dim + 4), rnd(M, kvh * dim + 4) * 1e-2, rnd(M, heads * vdim + 4) * (1e3 if case % 2 else 1.0)
        a = rnd(M, heads + 3) if kind == "state_space" else rnd(M, 8)
        out = torch.empty((M, heads * vdim), dtype=torch.float32, device=DEV)
        more = dict(heads=heads, dim=dim, vdim=vdim, state_offset=8, chunked=True)
        qd, kd, vd = ((t.double()[:, 4 * i:4 * i + n].view(M, -1, s)) for t, i, n, s in
                      ((q, 1, kvh * dim, dim), (k, 0, kvh * dim, dim), (v, 1, heads * vdim, vdim)))
        qd, kd = qd.repeat_interleave(heads // kvh, 1), kd.repeat_interleave(heads // kvh, 1)
        extra = None
        if kind == "state_space":
            ks.state_space_scan((q, 4), (k, 0), (v, 4), (a, 2), out, batch, state, kv_heads=kvh, a_log=a_log, dt_bias=dt, skip=skip, **more)
            step_size = torch.nn.functional.softplus(a.double()[:, 2:2 + heads] + dt.double())
            w = torch.exp(-torch.exp(a_log.double()) * step_size)[:, :, None, None]
            kd = kd * step_size[:, :, None]
        elif kind == "memory":
            z = rnd(M, heads * dim)
            w = torch.exp(-torch.exp(z.double() + w0.double())).view(M, heads, 1, dim)
            ks.decay_scan((q, 4), (k, 0), (v, 4), z, out, batch, state, w0=w0, u=u, **more)
            extra = u.double().view(heads, dim)
        else:
            decays = torch.empty((M, heads * dim), device=DEV)
            ks.gated_linear_scan((q, 4), (k, 0), (v, 4), (a, 1), decays, out, batch, state, a2=a2, a2_bias=a2_bias, tau=4.0, q_scale=0.3, **more)
            w = torch.sigmoid(a.double()[:, 1:7] @ a2.double() + a2_bias.double()).pow(0.25).view(M, heads, 1, dim)
            qd = qd * 0.3
        off = 0
        for s, n in enumerate(counts):
            part = slice(off, off + n)
            ref, carried[s] = scan_reference(kind, qd[part], kd[part], vd[part], w[part], extra, carried[s])
            if kind == "state_space":
                ref = ref + skip.double()[:, None] * vd[part]
            near(out[part].view(n, heads, vdim), ref, f"step {step}, segment {s}")
            got = state[slots[s], 8:8 + size].view(heads, vdim, dim4)
            near(got[:, :, :dim], carried[s], f"step {step}, state of segment {s}")
            assert not got[:, :, dim:].any()
            off += n


@pytest.mark.parametrize("kind", ["state_space", "memory"])
def test_scans_with_an_infinity_are_walked_token_by_token(kind):
    heads, dim, vdim, counts = 2, 64, 32, [70, 40]
    ks = kernels(torch.bfloat16)
    g = torch.Generator().manual_seed(6)
    rnd = lambda *s: torch.randn(s, generator=g).to(DEV)
    batch, M = step_batch(counts, [0, 1], True)
    q, k, v, a = rnd(M, heads * dim), rnd(M, heads * dim), rnd(M, heads * vdim), rnd(M, heads)
    v[50, 20] = float("inf")                                              # head 0, second group of 16 columns, first segment
    z, par, chan = rnd(M, heads * dim), rnd(heads), rnd(heads * dim)
    outs, states = [], []
    for chunked in (True, False):
        state = torch.zeros((2, heads * dim * vdim), device=DEV)
        out = torch.empty((M, heads * vdim), device=DEV)
        if kind == "state_space":
            ks.state_space_scan((q, 0), (k, 0), (v, 0), (a, 0), out, batch, state, heads=heads, kv_heads=heads, dim=dim, vdim=vdim, a_log=par,
                                dt_bias=par, skip=par, chunked=chunked)
        else:
            ks.decay_scan((q, 0), (k, 0), (v, 0), z.clone(), out, batch, state, heads=heads, dim=dim, vdim=vdim, w0=chan, u=chan, chunked=chunked)
        outs.append(out)
        states.append(state)
    torch.testing.assert_close(outs[0][:70, 16:32], outs[1][:70, 16:32], rtol=TOL, atol=0, equal_nan=True)
    assert not torch.isfinite(outs[0][50:70, 20]).any()
    near(outs[0][:50], outs[1][:50].double(), "before the infinity")
    near(outs[0][:, vdim:], outs[1][:, vdim:].double(), "the other head")
    near(outs[0][:, :16], outs[1][:, :16].double(), "the other columns")
    torch.testing.assert_close(states[0], states[1], rtol=1e-3, atol=1e-3, equal_nan=True)


# ---------------------------------------------------------------------------- the matrix memory
MEMORY = [
    (1, 256, 64, [(64, 1), (33, 31), (1, 95)]),
    (3, 20, 12, [(32, 17), (15, 16), (129, 2)]),
    (2, 128, 70, [(31, 65), (16, 1)]),
    (2, 200, 33, [(250, 97)]),
    (8, 64, 96, [(40, 33), (70, 1), (18, 9)]),
]


@pytest.mark.parametrize("case", range(len(MEMORY)))
@pytest.mark.parametrize("cap", [5.0, 30.0])
def test_matrix_memory_in_chunks(cap, case):
    heads, dim, vdim, segs = MEMORY[case]
    ks = kernels(torch.bfloat16)
    g = torch.Generator().manual_seed(90 + case)
    rnd = lambda *s: torch.randn(s, generator=g).to(DEV)
    size = ks.mlstm_state_size(dim, vdim)
    slots = torch.randperm(len(segs) + 2, generator=g)[:len(segs)].tolist()
    state = rnd(len(segs) + 2, heads, size)
    state[slots] = 0.0
    bi, bf = rnd(heads), rnd(heads) + 3.0
    cols = (1, 1 + heads * dim, 3 + 2 * heads * dim, 3 + 2 * heads * dim + heads * vdim, 4 + 2 * heads * dim + heads * (vdim + 1))
    carried = [[torch.zeros(s, dtype=torch.float64, device=DEV) for s in ((heads, dim, vdim), (heads, dim), (heads,))] for _ in segs]
    for step in range(2):
        counts = [s[step] for s in segs]
        batch, M = step_batch(counts, slots, step == 0)
        x = rnd(M, cols[4] + heads + 1)
        x[:, cols[3]:] *= cap
        x[:, cols[2]:cols[3]] *= 1e3 if case % 2 else 1e-2
        out = torch.empty((M, heads * vdim), dtype=torch.float32, device=DEV)
        ks.mlstm_scan(x, out, batch, state, heads=heads, dim=dim, vdim=vdim, gate_cap=cap, q_scale=dim ** -0.5, columns=cols, i_bias=bi,
                      f_bias=bf, chunked=True)
        xd, off = x.double(), 0
        q, k = xd[:, cols[0]:cols[0] + heads * dim].view(M, heads, dim) * dim ** -0.5, xd[:, cols[1]:cols[1] + heads * dim].view(M, heads, dim)
        v = xd[:, cols[2]:cols[2] + heads * vdim].view(M, heads, vdim)
        gi = cap * torch.tanh((xd[:, cols[3]:cols[3] + heads] + bi.double()) / cap)
        gf = torch.nn.functional.logsigmoid(cap * torch.tanh((xd[:, cols[4]:cols[4] + heads] + bf.double()) / cap))
        for s, n in enumerate(counts):
            S, nn, m = carried[s]
            ref = torch.zeros((n, heads, vdim), dtype=torch.float64, device=DEV)
            for t in range(off, off + n):
                new = torch.maximum(gf[t] + m, gi[t])
                keep, take = torch.exp(gf[t] + m - new)[:, None], torch.exp(gi[t] - new)[:, None] * k[t]
                m = new
                S, nn = keep[:, :, None] * S + take[:, :, None] * v[t][:, None, :], keep * nn + take
                den = torch.maximum((nn * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                ref[t - off] = torch.einsum("hkv,hk->hv", S, q[t]) / den[:, None]
            carried[s] = [S, nn, m]
            got = out[off:off + n].view(n, heads, vdim)
            # (a denominator near its floor of exp(-m) is a small difference of large sums: the tokens' own scale)
            near(got, ref, f"step {step}, segment {s}", 1e-4)
            st = state[slots[s]]
            near(st[:, :dim * vdim].view(heads, dim, vdim), S, f"step {step}, state of segment {s}")
            for c in range(-(-vdim // 32)):
                copy = st[:, dim * vdim + c * (-(-(dim + 1) // 4) * 4):][:, :dim + 1]
                near(copy[:, :dim], nn, "n")
                near(copy[:, dim], m, "m")
            off += n


def test_matrix_memory_with_an_infinity_is_walked_token_by_token():
    heads, dim, vdim, counts = 2, 64, 64, [70, 40]
    ks = kernels(torch.bfloat16)
    g = torch.Generator().manual_seed(7)
    batch, M = step_batch(counts, [0, 1], True)
    cols = (0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim, 2 * heads * dim + heads * vdim + heads)
    x = torch.randn((M, cols[4] + heads), generator=g).to(DEV)
    x[50, cols[2] + 40] = float("inf")
    outs, states = [], []
    for chunked in (True, False):
        state = torch.zeros((2, heads, ks.mlstm_state_size(dim, vdim)), device=DEV)
        out = torch.empty((M, heads * vdim), device=DEV)
        ks.mlstm_scan(x, out, batch, state, heads=heads, dim=dim, vdim=vdim, gate_cap=5.0, q_scale=0.1, columns=cols,
                      i_bias=torch.zeros(heads, device=DEV), f_bias=torch.zeros(heads, device=DEV), chunked=chunked)
        outs.append(out)
        states.append(state)
    torch.testing.assert_close(outs[0][:70, 32:64], outs[1][:70, 32:64], rtol=TOL, atol=0, equal_nan=True)
    near(outs[0][:50], outs[1][:50].double(), "before the infinity", 1e-4)
    near(outs[0][:, vdim:], outs[1][:, vdim:].double(), "the other head", 1e-4)
    near(outs[0][:, :32], outs[1][:, :32].double(), "the other block of columns", 1e-4)
    torch.testing.assert_close(states[0], states[1], rtol=1e-3, atol=1e-3, equal_nan=True)


def test_scan_and_memory_entry_points_refuse_malformed_calls():
    from spite_b200.kernels import build
    from spite_b200.kernels.cuda import MlstmParams, ScanParams
    scan, rec = build.load("scan"), build.load("recurrent")
    for f in (scan.spite_scan_chunk_bytes, rec.spite_mlstm_tiles_bytes):
        f.restype = C.c_longlong
    assert scan.spite_scan_chunk_bytes(0, 129, 8, 1, 1, 1, 1) == -2 and scan.spite_scan_chunk_bytes(1, 8, 0, 1, 1, 1, 1) == -1
    assert rec.spite_mlstm_tiles_bytes(257, 8, 1, 1, 1) == -2 and rec.spite_mlstm_tiles_bytes(8, 8, 0, 1, 1) == -1
    t = torch.zeros(1 << 16, device=DEV)
    at, stride = t.data_ptr(), C.c_longlong(16)
    vp = C.c_void_p
    a = dict.fromkeys(("q", "k", "v", "scalars", "out", "state", "cu_seqlens", "slots"), at)
    a.update(q_stride=16, k_stride=16, v_stride=16, out_stride=16, slot_stride=256, n_segments=1, n_tokens=4, heads=1, kv_heads=1, dim=16, vdim=16,
             out_scale=1.0)

    def walks(scratch=at, chunks=1, least=1, **k):
        p, w = ScanParams(**dict(a, **k)), ScanParams(**dict(a, w=at, w_stride=k.get("dim", 16), **k))
        tail = (vp(scratch), chunks, least, None)
        return [scan.spite_state_space_scan_chunked(C.byref(p), vp(at), stride, vp(at), vp(at), *tail),
                scan.spite_decay_scan_chunked(C.byref(w), vp(at), vp(at), *tail),
                scan.spite_gated_linear_scan_chunked(C.byref(w), vp(at), stride, vp(at), vp(at), 4, C.c_float(2.0), *tail)]
    for bad in (dict(scratch=None), dict(scratch=at + 4), dict(chunks=0), dict(least=0), dict(heads=0), dict(vdim=0)):
        assert walks(**bad) == [-1] * 3, bad
    assert walks(dim=160, q_stride=160, k_stride=160, slot_stride=1 << 14) == [-2] * 3
    assert walks(n_segments=0) == [0] * 3 and walks(n_tokens=0) == [0] * 3
    m = dict.fromkeys(("proj", "out", "state", "cu_seqlens", "slots"), at)
    m.update(stride=200, q_col=0, k_col=16, v_col=32, i_col=48, f_col=49, head_stride=400, n_segments=1, heads=1, dim=16, vdim=16, gate_cap=1.0,
             q_scale=1.0)
    tiles = lambda scratch=at, chunks=1, least=1, **k: rec.spite_mlstm_scan_tiles(C.byref(MlstmParams(**dict(m, **k))), vp(scratch), chunks, least, None)
    assert tiles(scratch=None) == tiles(scratch=at + 4) == tiles(chunks=0) == tiles(least=0) == tiles(heads=0) == tiles(gate_cap=0.0) == -1
    assert tiles(dim=300, stride=1000, head_stride=1 << 14) == -2 and tiles(n_segments=0) == 0
    torch.cuda.synchronize()
    assert not t.any()


def test_a_wait_that_runs_out_in_the_delta_rule_is_reported_and_the_tokens_are_walked():
    """The first stage is announced 16 bytes more than its copies deliver, with waits of two milliseconds: every block of the walk in
    chunks gives up, says so, and leaves its columns to the walk token by token."""
    heads, dim, vdim, n = 2, 64, 32, 70
    ks = kernels(torch.bfloat16)
    g = torch.Generator().manual_seed(8)
    batch, M = step_batch([n], [0], True)
    cols = (0, dim * heads, 2 * dim * heads, 2 * dim * heads + heads * vdim, 2 * dim * heads + heads * vdim + heads)
    x = torch.randn((M, cols[4] + heads), generator=g).to(DEV)
    zero = torch.zeros(heads, device=DEV)

    def run(chunked):
        state, out = torch.zeros((1, heads * dim * vdim), device=DEV), torch.empty((M, heads * vdim), device=DEV)
        ks.delta_scan(x, out, batch, state, heads=heads, kv_heads=heads, dim=dim, vdim=vdim, columns=cols, a_log=zero, dt_bias=zero, q_scale=1.0,
                      chunked=chunked)
        torch.cuda.synchronize()
        return out, state
    want = run(False)
    assert ks.errors() == {}
    ks.configure_waits("delta", limit_cycles=4_000_000, extra_tx=16)
    try:
        got = run(True)
    finally:
        ks.configure_waits("delta")
    assert ks.errors() == {"delta": 2} and ks.errors() == {}
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    near(run(True)[0], want[0].double(), "with the default waits")
    assert ks.errors() == {}


# ---------------------------------------------------------------------------- the order of what warps do
def walks(kind, ks, g, counts, heads, dim, vdim, scale=lambda name, t: t):
    """A function that makes one pass of a walk in chunks over new states: () -> (outputs [M, heads * vdim], states).  `scale` may change
    the drawn q, k, v."""
    rnd = lambda *s: torch.randn(s, generator=g).to(DEV)
    batch, M = step_batch(counts, list(range(len(counts))), True)
    q, k, v = (scale(n, rnd(M, heads, w)).reshape(M, -1) for n, w in (("q", dim), ("k", dim), ("v", vdim)))
    a, b, par, z, chan = rnd(M, heads), rnd(M, heads), rnd(heads), rnd(M, heads * dim) - 2.0, rnd(heads * dim) - 1.0
    a2, wide = rnd(6, heads * dim), torch.cat([q, k, v, a, b], 1).contiguous()
    n, m = heads * dim, 2 * heads * dim + heads * vdim
    cols = (0, n, 2 * n, m, m + heads)

    def run(chunked=True):
        out = torch.empty((M, heads * vdim), device=DEV)
        shape = (heads, ks.mlstm_state_size(dim, vdim)) if kind == "matrix_memory" else (
            heads * (dim * vdim if kind == "delta" else ks.scan_state_size(dim, vdim)),)
        state = torch.zeros((len(counts),) + shape, device=DEV)
        more = dict(heads=heads, dim=dim, vdim=vdim, chunked=chunked)
        if kind == "matrix_memory":
            ks.mlstm_scan(wide, out, batch, state, gate_cap=8.0, q_scale=dim ** -0.5, columns=cols, i_bias=par, f_bias=par + 3.0, **more)
        elif kind == "delta":
            ks.delta_scan(wide, out, batch, state, kv_heads=heads, columns=cols, a_log=par, dt_bias=par, q_scale=dim ** -0.5, **more)
        elif kind == "state_space":
            ks.state_space_scan((q, 0), (k, 0), (v, 0), (a, 0), out, batch, state, kv_heads=heads, a_log=par, dt_bias=par - 3.0, skip=par, **more)
        elif kind == "decaying_memory":
            ks.decay_scan((q, 0), (k, 0), (v, 0), z.clone(), out, batch, state, w0=chan, u=chan, **more)
        else:
            ks.gated_linear_scan((q, 0), (k, 0), (v, 0), (wide, 0), torch.empty((M, n), device=DEV), out, batch, state, a2=a2, a2_bias=chan + 2.0,
                                 tau=8.0, q_scale=0.2, **more)
        return out, state

    def reference():
        """The same in float64, token by token: outputs [M, heads, vdim] and, per segment, the matrices [heads, vdim, dim]."""
        f = lambda t: t.double().view(M, heads, -1)
        qd, kd, vd, ad, bd, pd = f(q), f(k), f(v), a.double(), b.double(), par.double()
        outs, states, off = [], [], 0
        for n_tokens in counts:
            part = slice(off, off + n_tokens)
            off += n_tokens
            if kind == "delta":
                out, S = delta_reference(wide[part], cols, heads, heads, dim, vdim, par, par, dim ** -0.5,
                                         torch.zeros((heads, dim, vdim), dtype=torch.float64, device=DEV))
                S = S.transpose(1, 2)
            elif kind == "matrix_memory":
                out, S = memory_reference(qd[part] * dim ** -0.5, kd[part], vd[part], 8.0 * torch.tanh((ad[part] + pd) / 8.0),
                                          torch.nn.functional.logsigmoid(8.0 * torch.tanh((bd[part] + pd + 3.0) / 8.0)))
            else:
                S, qs, ks_, extra = torch.zeros((heads, vdim, dim), dtype=torch.float64, device=DEV), qd[part], kd[part], None
                if kind == "state_space":
                    step = torch.nn.functional.softplus(ad[part] + pd - 3.0)
                    w, ks_ = torch.exp(-torch.exp(pd) * step)[:, :, None, None], ks_ * step[:, :, None]
                elif kind == "decaying_memory":
                    w, extra = torch.exp(-torch.exp(z[part].double() + chan.double())).view(-1, heads, 1, dim), chan.double().view(heads, dim)
                else:
                    w = torch.sigmoid(wide[part, :6].double() @ a2.double() + chan.double() + 2.0).pow(0.125).view(-1, heads, 1, dim)
                    qs = qs * 0.2
                out, S = scan_reference("memory" if kind == "decaying_memory" else kind, qs, ks_, vd[part], w, extra, S)
                if kind == "state_space":
                    out = out + pd[:, None] * vd[part]
            outs.append(out)
            states.append(S)
        return torch.cat(outs), torch.stack(states)

    def matrices(state):
        """The matrices [segments, heads, vdim, dim] of the states."""
        if kind in ("matrix_memory", "delta"):
            return state.view(len(counts), heads, -1)[:, :, :dim * vdim].view(len(counts), heads, dim, vdim).transpose(2, 3)
        return state.view(len(counts), heads, vdim, dim)
    run.reference, run.matrices = reference, matrices
    return run


def memory_reference(q, k, v, gi, gf):
    T, H, _ = q.shape
    S, n, m, out = (torch.zeros(s, dtype=torch.float64, device=q.device) for s in ((H, v.shape[2], q.shape[2]), (H, q.shape[2]), (H,), v.shape))
    for t in range(T):
        new = torch.maximum(gf[t] + m, gi[t])
        keep, take = torch.exp(gf[t] + m - new)[:, None], torch.exp(gi[t] - new)[:, None] * k[t]
        m = new
        S, n = keep[:, :, None] * S + v[t][:, :, None] * take[:, None, :], keep * n + take
        out[t] = torch.einsum("hvk,hk->hv", S, q[t]) / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
    return out, S


KINDS = ["matrix_memory", "delta", "state_space", "decaying_memory", "linear_attention"]


@pytest.mark.parametrize("kind", KINDS)
def test_passes_of_the_same_input_are_the_same_bits(kind):
    """Many chunks, heads and segments of unequal length, alone and beside products on another stream that take multiprocessors and
    change the warps' pace: what a warp makes for others (sums, factors, scales) is ordered before their reads, whoever comes first."""
    ks = kernels(torch.bfloat16)
    dim = 256 if kind == "matrix_memory" else 128
    run = walks(kind, ks, torch.Generator().manual_seed(12), [517, 97, 260, 33, 1025], 8, dim, 256)
    want = run()
    assert torch.isfinite(want[0]).all()
    x, y = torch.randn((2048, 2048), device=DEV), torch.empty((2048, 2048), device=DEV)
    side = torch.cuda.Stream()
    for i in range(12):
        if i % 2:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                for _ in range(1 + i):
                    torch.mm(x, x, out=y)
        got = run()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), f"pass {i}"
    assert ks.errors() == {}


@pytest.mark.parametrize("kind", KINDS)
def test_a_block_that_gives_up_waits_for_its_first_chunk_before_it_leaves(kind):
    """The first chunk's stage is announced 16 bytes more than its copies deliver: the wait for it runs out, and the block waits for that
    stage's copies once more, with the same limit, since they could land in shared memory that is another block's by then."""
    limit, library = 8_000_000, {"matrix_memory": "recurrent", "delta": "delta"}.get(kind, "scan")
    ks = kernels(torch.bfloat16)
    run = walks(kind, ks, torch.Generator().manual_seed(13), [70, 150], 2, 64, 32)
    want = run(False)
    run()
    torch.cuda.synchronize()
    assert ks.errors() == {}
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ks.configure_waits(library, limit_cycles=limit, extra_tx=16)
    try:
        begin.record()
        got = run()
        end.record()
        torch.cuda.synchronize()
    finally:
        ks.configure_waits(library)
    assert ks.errors() == {library: 2} and ks.errors() == {}
    # two limits of 8 million clocks at 2.0 GHz at most (a single one and the tokens' walk take 4.1 to 5 ms)
    assert begin.elapsed_time(end) >= 2 * limit / 2.0e6
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    near(run()[0], want[0].double(), "with the default waits", 1e-4)
    assert ks.errors() == {}


# ---------------------------------------------------------------------------- numbers of very different size
@pytest.mark.parametrize("uneven", ["even", "columns", "tokens", "keys"])
@pytest.mark.parametrize("kind", KINDS)
def test_columns_tokens_and_keys_of_different_size_keep_their_bits(kind, uneven):
    """Value columns that differ by 10^12, tokens and keys by 10^6: every column, token and key is held as the walk token by token holds
    it.  The error against float64, relative to the largest element of the column, the token or the key's row of the state, is at most
    three times that walk's, plus 40 units of 2^-23 for the sums' other order (128 terms a product, a few products)."""
    heads, dim, vdim, counts = 2, 128, 64, [100, 300]
    ks = kernels(torch.bfloat16)
    g = torch.Generator().manual_seed(21)
    r = lambda n, span: 10.0 ** ((torch.rand(n, generator=g) * 2.0 - 1.0) * span).to(DEV)
    by_column, by_key, M = r(vdim, 6.0), r(dim, 3.0), sum(counts)
    by_token = {n: r(M, 3.0)[:, None, None] for n in "qkv"}

    def scale(name, t):
        if uneven == "tokens":
            return t * by_token[name]
        if uneven == "columns" and name == "v":
            return t * by_column
        # (a key's part of every q . k stays what it was, while q, k and the state differ from key to key)
        return t * by_key if uneven == "keys" and name == "q" else t / by_key if uneven == "keys" and name == "k" else t
    run = walks(kind, ks, g, counts, heads, dim, vdim, scale)
    want, want_state = run.reference()

    def errors(chunked):
        out, state = run(chunked)
        e, es = (out.double().view_as(want) - want).abs(), (run.matrices(state).double() - want_state).abs()
        out_axes = {"tokens": 2}.get(uneven, 0)                          # the axis over which the largest element is looked for
        state_axes = {"keys": 2}.get(uneven, 3)
        rel = lambda e, w, axis: float((e.amax(axis) / w.abs().amax(axis)).max())
        return rel(e, want, out_axes), rel(es, want_state, state_axes)
    chunks, tokens = errors(True), errors(False)
    print(f"{kind} {uneven}: output {chunks[0]:.2e} ({tokens[0]:.2e} token by token), state {chunks[1]:.2e} ({tokens[1]:.2e})")
    for c, t in zip(chunks, tokens):
        assert c <= 3.0 * t + 40 * 2.0**-23


# ---------------------------------------------------------------------------- working memory
class _Fewer:
    """A kernel library whose walks in chunks are told of `n` chunks."""

    def __init__(self, lib, n):
        self.lib, self.n = lib, n

    def __getattr__(self, name):
        f = getattr(self.lib, name)
        return (lambda *a: f(*a[:-3], self.n, *a[-2:])) if name.endswith(("_chunked", "_tiles")) else f


@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 7])
@pytest.mark.parametrize("kind", KINDS)
def test_working_memory_for_fewer_chunks_than_the_step_has(kind, n):
    """Segments that a caller's working memory has no place for go token by token, and nothing is written behind it."""
    counts, heads, dim, vdim = [40, 70, 3, 64], 2, 64, 32
    library = {"matrix_memory": "recurrent", "delta": "delta"}.get(kind, "scan")
    ks = kernels(torch.bfloat16)
    run = walks(kind, ks, torch.Generator().manual_seed(14), counts, heads, dim, vdim)
    want, whole = run(False), run()
    buffers = []

    def scratch(library, query, *sizes):
        f = getattr(ks._lib(library).lib, query)
        f.restype = C.c_longlong
        need = f(*(int(x) for x in sizes[:-2]), n, int(sizes[-1]))
        buffers.append((torch.full((need + (1 << 16),), 0x5a, dtype=torch.uint8, device=DEV), need))
        return buffers[-1][0]
    ks._chunk_scratch = scratch
    ks._libs[library] = _Fewer(ks._lib(library), n)
    out, state = run()
    # (segments of fewer than 32 tokens, 8 in the matrix memory, have no chunks)
    at, off = 0, 0
    for s, tokens in enumerate(counts):
        chunks = -(-tokens // 32)
        part = slice(off, off + tokens)
        off += tokens
        ref = whole if tokens >= 32 and at + chunks <= n else want
        assert torch.equal(out[part], ref[0][part]) and torch.equal(state[s], ref[1][s]), f"segment {s}"
        at += chunks if tokens >= 32 else 0
    assert buffers and all(bool((b[need:] == 0x5a).all()) for b, need in buffers)


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("kind", KINDS)
def test_decode_tokens_beside_portions_take_no_chunks(kind, known):
    """Portions among many decoded tokens: the tokens' rows are the walk token by token's, the portions' the walk in chunks' alone, and
    working memory is asked for the portions only.  `known`: the entry points are told how many portions there are."""
    counts, heads, dim, vdim = [1] * 40 + [70] + [1] * 33 + [32, 1, 200] + [2] * 3, 2, 64, 48
    ks = kernels(torch.bfloat16)
    ks.memory_min_tokens = 32
    run = walks(kind, ks, torch.Generator().manual_seed(15), counts, heads, dim, vdim)
    asked, inner, of_batch = [], ks._chunk_scratch, ks._long_segments

    def scratch(library, query, *sizes):
        asked.append(sizes[-2])
        return inner(library, query, *sizes)
    ks._chunk_scratch = scratch
    if not known:
        ks._long_segments = lambda batch, least: (0, of_batch(batch, least)[1])
    want, got = run(False), run()
    assert asked == [3 + 1 + 7]
    off = 0
    for s, n in enumerate(counts):
        part = slice(off, off + n)
        off += n
        if n < 32:
            assert torch.equal(got[0][part], want[0][part]) and torch.equal(got[1][s], want[1][s]), f"segment {s}"
        else:
            near(got[0][part], want[0][part].double(), f"segment {s}", 1e-4)
            near(got[1][s], want[1][s].double(), f"state of segment {s}", 1e-4)
    assert ks.errors() == {}


@pytest.mark.parametrize("dim", [40, 100, 200])
@pytest.mark.parametrize("kind", KINDS)
def test_calls_beyond_the_limit_of_working_memory(kind, dim):
    """The matrix memory goes in chunks on the float32 units, the other walks token by token."""
    if kind != "matrix_memory" and dim > 128:
        pytest.skip("no walk in chunks: always token by token")
    ks = kernels(torch.bfloat16)
    ks.chunk_scratch_limit = 1 << 10
    library = {"matrix_memory": "recurrent", "delta": "delta"}.get(kind, "scan")
    run = walks(kind, ks, torch.Generator().manual_seed(16), [70, 33, 1], 2, dim, 40)
    want, want_state = run.reference()
    before = ks.launches_by_library[library]
    out, state = run()
    assert ks.launches_by_library[library] == before + 2
    near(out.view_as(want), want, "outputs", 1e-4)
    near(run.matrices(state), want_state, "states")
    if kind != "matrix_memory":
        tokens = run(False)
        assert torch.equal(out, tokens[0]) and torch.equal(state, tokens[1])


# (walk, heads, segments, in chunks): a portion beside decode tokens whose states hide the token walk's chain goes token by token
ROUTES = [("delta", 16, [40], True), ("delta", 16, [39], False), ("delta", 16, [72] + [1] * 16, True), ("delta", 16, [72] + [1] * 48, False),
          ("delta", 16, [1] * 100 + [256], True), ("state_space", 64, [192], True), ("state_space", 64, [191], False),
          ("state_space", 64, [256] + [1] * 16, False), ("state_space", 64, [512] + [1] * 16, True), ("linear_attention", 32, [384], True),
          ("linear_attention", 16, [384], False), ("linear_attention", 16, [300, 384], True), ("linear_attention", 32, [512] + [1] * 64, False),
          ("decaying_memory", 8, [2048], False), ("matrix_memory", 2, [8], True), ("matrix_memory", 2, [7], False),
          ("matrix_memory", 2, [1] * 50 + [9], True)]


@pytest.mark.parametrize("case", range(len(ROUTES)))
def test_which_steps_go_in_chunks_where_the_caller_leaves_it_open(case):
    kind, heads, counts, in_chunks = ROUTES[case]
    ks, exact = kernels(torch.bfloat16), kernels(torch.float32)
    library = {"matrix_memory": "recurrent", "delta": "delta"}.get(kind, "scan")
    for k, want in ((ks, in_chunks), (exact, False)):
        run = walks(kind, k, torch.Generator().manual_seed(17), counts, heads, 32, 16)
        before = k.launches_by_library[library]
        out, state = run(None)
        assert k.launches_by_library[library] - before == (1 if library == "recurrent" else 2) + want * (
            2 if kind in ("matrix_memory", "linear_attention") else 1)
        forced = run(want)
        assert torch.equal(out, forced[0]) and torch.equal(state, forced[1])
