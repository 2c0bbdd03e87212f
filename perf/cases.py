"""Workloads by which the engine's speed is followed: layers of the served designs in prompts and in decode steps, a
feed-forward of every kind, whole requests through the engine, and sampling.

A case names a kind of work (`kind`) and its sizes; layer sizes are those of the benchmark configurations (`bench.py`) or a
part of them.  `prepare` builds what a program keeps (weights, cache, captured step) and draws the inputs, `run` is one pass
through the parts, the engine or the sampler, `exact` the same in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import random

import torch

from spite_b200.cache import LayerCache, Window
from spite_b200.config import PartSpec, config_from_dict
from spite_b200.engine import Engine, Model
from spite_b200.engine.batch import Segment, build_step_batch
from spite_b200.kernels.cuda import CudaKernels
from spite_b200.parts import BuildContext, build_part
from spite_b200.sampling.sampler import Sampler, SampleRow, SamplingParams

DEV = "cuda:0"
PAGE = 64


def listed():
    return [
        # a late portion of a long prompt through an attention layer of Llama-4-Scout's sizes, one request
        dict(name="attention_prompt", kind="attention", width=5120, heads=40, kv_heads=8, requests=1, tokens=2048, context=8192),
        # the same layer in a captured decode step of eight requests whose contexts differ
        dict(name="attention_decode", kind="attention", width=5120, heads=40, kv_heads=8, requests=8, tokens=8, context=8192),
        # a matrix memory (xLSTM) over one prompt that fills the step's token budget
        dict(name="matrix_memory_prompt", kind="matrix_memory", width=4096, requests=1, tokens=2048),
        # a gated delta rule over the prompts of three requests of unequal, odd lengths in one step
        dict(name="delta_prompts", kind="delta", width=2048, requests=3, tokens=1999),
        # a state space (Mamba-2) over one prompt that fills the step's token budget
        dict(name="state_space_prompt", kind="state_space", width=4096, requests=1, tokens=2048),
        # gated linear attention over the prompts of five requests in one step
        dict(name="linear_attention_prompts", kind="linear_attention", width=4096, requests=5, tokens=2048),
        # a short prompt: the smallest step that is not a decode step, through a state space of the small width
        dict(name="state_space_short", kind="state_space", width=2048, requests=1, tokens=67),
        # the experts of a Llama-4-Scout layer, and the shared one, on the tokens of a prompt
        dict(name="experts_prompt", kind="experts_top1", width=5120, experts=16, inner=8192, tokens=1500),
        # experts chosen by softmax, two a token, in a captured decode step of eight requests
        dict(name="experts_decode", kind="experts_top2", width=2048, experts=32, inner=1024, tokens=8),
        # one request through the engine: a prompt of a few hundred tokens and 16 decode steps
        dict(name="request_alone", kind="requests", width=2048, requests=1, prompt=301, steps=16),
        # a full house of short requests through the engine: mostly decode steps
        dict(name="requests_many", kind="requests", width=2048, requests=24, prompt=24, steps=16),
        # the next tokens of 32 requests by temperature, top-p and repetition penalty over Llama 4's vocabulary
        dict(name="sampling", kind="sampling", rows=32, vocab=202048),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["attention", "attention", "matrix_memory", "delta", "delta", "state_space", "state_space", "linear_attention",
                       "experts_top1", "experts_top2", "requests", "sampling"])
    if kind == "attention":
        width = rng.choice([2048, 4096, 5120])
        c = dict(kind=kind, width=width, heads=width // 128, kv_heads=width // 128 // rng.choice([4, 4, 8] if width != 5120 else [5]))
        context = log(150, 8192)
        if rng.random() < 0.5:
            n = log(1, 12)
            return dict(c, requests=n, tokens=n, context=context)
        n = rng.randint(1, 3)
        return dict(c, requests=n, tokens=max(2 * n, min(log(17, 2048), n * context)), context=context)
    if kind in ("matrix_memory", "delta", "state_space", "linear_attention"):
        tokens = log(17, 2048)
        return dict(kind=kind, width=rng.choice([2048, 4096]), requests=min(rng.randint(1, 6), tokens // 8), tokens=tokens)
    if kind == "experts_top1":
        return dict(kind=kind, width=rng.choice([2048, 4096, 5120]), experts=rng.choice([8, 16]), inner=rng.choice([2048, 4096]),
                    tokens=log(40, 1500))
    if kind == "experts_top2":
        return dict(kind=kind, width=rng.choice([2048, 4096]), experts=rng.choice([16, 32]), inner=rng.choice([1024, 2048]), tokens=log(1, 32))
    if kind == "requests":
        return dict(kind=kind, width=rng.choice([1024, 2048]), requests=rng.randint(1, 12), prompt=log(9, 200), steps=rng.randint(4, 16))
    return dict(kind=kind, rows=log(1, 32), vocab=rng.choice([32768, 65536, 202048]))


# ------------------------------------------------------------------ inputs
class _Draws:
    """Tensors on the device from a seed, one after another."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 17)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=self.g)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(low, high, generator=self.g)


def _lengths(total, parts, least=1):
    """`total` tokens in `parts` unequal shares of at least `least`, the same for every seed."""
    r = random.Random(total * 31 + parts)
    w = [r.uniform(0.4, 1.6) for _ in range(parts)]
    n = [max(least, int(total * x / sum(w))) for x in w]
    n[0] += total - sum(n)
    return n


def _segments(case):
    """(first position, tokens) of every request of the step."""
    if case["kind"] != "attention":
        return [(0, n) for n in _lengths(case["tokens"], case["requests"])]
    if case["tokens"] == case["requests"]:
        r = random.Random(case["context"])
        ends = [case["context"]] + [r.randint(case["context"] // 4 + 1, case["context"]) for _ in range(case["requests"] - 1)]
        return [(e - 1, 1) for e in ends]
    return [(max(0, case["context"] - n), n) for n in _lengths(case["tokens"], case["requests"], 2)]


def _batch(segments):
    segs, tables, offset, page = [], [], 0, 0
    for i, (start, n) in enumerate(segments):
        segs.append(Segment(i, i, start, n, offset, start == 0))
        pages = -(-(start + n) // PAGE)
        tables.append(list(range(page, page + pages)))
        offset, page = offset + n, page + pages
    return build_step_batch(segs, [[0] * n for _, n in segments], [[] for _ in segments], [tables], DEV), page


def _layer(case):
    """The part of a layer case, as a model's plan names it."""
    d = case["width"]
    return {
        "attention": lambda: ("mixer", PartSpec("paged_attention", dict(
            hidden_size=d, num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=128, window=("chunk", 8192), qk_norm_eps=1e-5,
            position=PartSpec("rotary_interleaved", dict(head_dim=128, theta=500000.0))))),
        "matrix_memory": lambda: ("mixer", PartSpec("mlstm", dict(
            hidden_size=d, num_heads=8, head_dim=d // 16, value_dim=d // 8, gate_cap=10.0, norm_eps=1e-5))),
        "delta": lambda: ("mixer", PartSpec("gated_delta", dict(
            hidden_size=d, num_heads=d // 128, num_kv_heads=d // 256, head_dim=128, value_dim=128, conv_taps=4, norm_eps=1e-6))),
        "state_space": lambda: ("mixer", PartSpec("state_space", dict(
            hidden_size=d, num_heads=d // 32, value_dim=64, state_size=128, groups=1, conv_taps=4, norm_groups=1, norm_eps=1e-6))),
        "linear_attention": lambda: ("mixer", PartSpec("gated_linear_attention", dict(
            hidden_size=d, num_heads=d // 128, head_dim=64, value_dim=128, decay_rank=16, tau=16.0, norm_eps=1e-6))),
        "experts_top1": lambda: ("feed_forward", PartSpec("moe_sigmoid_prescaled", dict(
            hidden_size=d, num_experts=case["experts"], top_k=1, expert_size=case["inner"], shared_size=case["inner"]))),
        "experts_top2": lambda: ("feed_forward", PartSpec("moe_softmax_topk", dict(
            hidden_size=d, num_experts=case["experts"], top_k=2, expert_size=case["inner"]))),
    }[case["kind"]]()


def _params(case, r):
    """A layer's parameters: matrices N(0, 0.02), the recurrences' constants over the ranges such models are started with."""
    d, kind, f32 = case["width"], case["kind"], torch.float32
    w = lambda *shape: r.normal(*shape, std=0.02)
    if kind == "attention":
        n, m = case["heads"] * 128, case["kv_heads"] * 128
        return dict(q_proj=w(n, d), k_proj=w(m, d), v_proj=w(m, d), o_proj=w(d, n))
    if kind == "matrix_memory":
        H, dk, dv = 8, d // 16, d // 8
        return dict(q_proj=w(H * dk, d), k_proj=w(H * dk, d), v_proj=w(H * dv, d), gate_proj=w(H * dv, d), o_proj=w(d, H * dv),
                    norm=r.uniform(H * dv, low=0.8, high=1.2), igate_proj=w(H, d), igate_bias=r.uniform(H, low=-3.0, high=0.0),
                    fgate_proj=w(H, d), fgate_bias=r.uniform(H, low=3.0, high=6.0))
    steps = lambda n: torch.log(torch.expm1(torch.exp(r.uniform(n, low=math.log(0.001), high=math.log(0.1)))))
    if kind == "delta":
        H, G, dk, dv = d // 128, d // 256, 128, 128
        taps = lambda n: r.uniform(n, 4, low=-0.5, high=0.5)
        return dict(q_proj=w(G * dk, d), k_proj=w(G * dk, d), v_proj=w(H * dv, d), q_conv=taps(G * dk), k_conv=taps(G * dk),
                    v_conv=taps(H * dv), beta_proj=w(H, d), decay_proj=w(H, d), a_log=torch.log(r.uniform(H, low=1.0, high=16.0)),
                    dt_bias=steps(H), gate_proj=w(H * dv, d), norm=r.uniform(dv, low=0.8, high=1.2), o_proj=w(d, H * dv))
    if kind == "state_space":
        H, n, N = d // 32, d * 2, 128
        return dict(in_proj=w(2 * n + 2 * N + H, d), conv=r.uniform(n + 2 * N, 4, low=-0.5, high=0.5),
                    conv_bias=r.uniform(n + 2 * N, low=-0.5, high=0.5), dt_bias=steps(H), a_log=torch.log(r.uniform(H, low=1.0, high=16.0)),
                    skip=torch.ones(H, device=DEV), norm=r.uniform(n, low=0.8, high=1.2), o_proj=w(d, n))
    if kind == "linear_attention":
        H, nk, nv = d // 128, d // 2, d
        return dict(q_proj=w(nk, d), k_proj=w(nk, d), v_proj=w(nv, d), gate_proj=w(nv, d), decay_in=w(16, d),
                    decay_out=r.normal(nk, 16, std=0.1), decay_bias=r.uniform(nk, low=-1.0, high=1.0),
                    norm=r.uniform(128, low=0.8, high=1.2), o_proj=w(d, nv))
    E, f = case["experts"], case["inner"]
    if kind == "experts_top1":
        return dict(router=w(E, d).to(f32), experts_gate_up=w(E, 2 * f, d), experts_down=w(E, d, f), shared_gate_proj=w(f, d),
                    shared_up_proj=w(f, d), shared_down_proj=w(d, f))
    return dict(router=w(E, d).to(f32), experts_gate=w(E, f, d), experts_up=w(E, f, d), experts_down=w(E, d, f))


def _model_config(case):
    """Two matrix memories and two attention layers, of which one reads the other's keys, dense feed-forwards behind them."""
    d = case["width"]
    mem = {"type": "mlstm", "mixer": {"heads": 8, "dim": d // 16, "vdim": d // 8, "gate_cap": 10.0}, "mlp": None}
    att = lambda src: {"type": "attention", "mlp": {"kind": "dense", "ff": 4 * d}, "mixer": dict(
        {"heads": d // 128, "kv_heads": d // 512, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 8192},
         "rot": {"base": 500000.0, "dims": 64}}, **({} if src is None else {"kv_from": src}))}
    return {"architecture": "Paposun", "vocab": 32768, "width": d, "max_positions": 8192, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
            "logit_scale": 0.5, "layers": [mem, att(None), att(1), mem]}


def _model_params(case, seed):
    r, d, n, m, v = _Draws(seed), case["width"], case["width"], case["width"] // 4, case["width"]
    w = lambda *shape: r.normal(*shape, std=0.02)
    gain = lambda k: r.uniform(k, low=0.8, high=1.2)
    out = {"embed.weight": r.normal(32768, d, std=0.5), "final_norm.weight": gain(d)}
    for i in range(4):
        at = f"layers.{i}."
        out.update({at + "mixer_norm.weight": gain(d), at + "mixer_out_norm.weight": gain(d)})
        if i in (0, 3):
            out.update({at + "mixer." + k: t for k, t in _params(dict(case, kind="matrix_memory"), r).items()})
            continue
        names = ["q", "k", "v"] if i == 1 else ["q"]
        for s in names:
            out[at + f"mixer.{s}_proj"], out[at + f"mixer.{s}_bias"] = w(n if s == "q" else m, d), r.uniform(n if s == "q" else m, low=-0.1, high=0.1)
        out.update({at + "mixer.out_gate_proj": w(v, d), at + "mixer.o_proj": w(d, v), at + "mixer.o_bias": r.uniform(d, low=-0.1, high=0.1),
                    at + "ffn_norm.weight": gain(d), at + "ffn_out_norm.weight": gain(d), at + "ffn.up_proj": w(4 * d, d),
                    at + "ffn.down_proj": w(d, 4 * d)})
    return out


def _sequences(case, seed):
    """Every request's prompt and the tokens that its decode steps are given."""
    r = random.Random(seed * 7919 + 5)
    lengths = _lengths(case["prompt"] * case["requests"], case["requests"], 2)
    return [([r.randrange(32768) for _ in range(n)], [r.randrange(32768) for _ in range(case["steps"])]) for n in lengths]


# ------------------------------------------------------------------ a pass
def prepare(case, seed):
    kind = case["kind"]
    if kind == "sampling":
        r, host = _Draws(seed), random.Random(seed)
        k = CudaKernels(torch.float32, DEV)
        rows = [SampleRow(SamplingParams(temperature=host.uniform(0.6, 1.0), top_p=host.choice([0.9, 0.95]), top_k=host.choice([0, 40]),
                                         repetition_penalty=1.1, repeat_last_n=64),
                          [host.randrange(case["vocab"]) for _ in range(host.randint(1, 200))], host.getrandbits(64))
                for _ in range(case["rows"])]
        return dict(kind=kind, sampler=Sampler(k), rows=rows, logits=r.normal(case["rows"], case["vocab"], std=2.5, dtype=torch.float32))
    if kind == "requests":
        model = Model.from_config(config_from_dict(_model_config(case)), dtype="bfloat16", device=DEV).load_params(_model_params(case, seed))
        seqs = _sequences(case, seed)
        longest = max(len(p) for p, _ in seqs) + case["steps"]
        engine = Engine(model, cache_tokens=case["requests"] * (longest + PAGE), page_size=PAGE, max_requests=case["requests"], max_positions=8192)
        return dict(kind=kind, engine=engine, seqs=seqs, steps=case["steps"])
    r = _Draws(seed)
    family, spec = _layer(case)
    ctx = BuildContext(CudaKernels(torch.bfloat16, DEV), torch.bfloat16, torch.device(DEV))
    part = build_part(family, spec, ctx)
    part.bind(_params(case, r))
    x = r.normal(case["tokens"], case["width"])
    s = dict(kind=kind, part=part, x=x, y=torch.empty((case["tokens"], case["width"]), dtype=torch.float32, device=DEV))
    if family == "feed_forward":
        s["batch"], s["cache"] = None, None
    else:
        s["batch"], pages = _batch(_segments(case))
        kv = state = None
        if kind == "attention":
            kv = r.normal(2, pages, case["kv_heads"], PAGE, 128)
        else:
            state = torch.zeros((case["requests"],) + tuple(part.cache_request()[1].shape), dtype=torch.float32, device=DEV)
        s["cache"] = LayerCache(0 if kv is not None else None, kv, state, PAGE, True)
    if case["tokens"] <= 32 and (family == "feed_forward" or (kind == "attention" and case["tokens"] == case["requests"])):
        # decode steps are captured and replayed, as the engine does
        side = torch.cuda.Stream(device=DEV)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _forward(s)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _forward(s)
        s["graph"] = graph
    return s


def _forward(s):
    if s["kind"] == "experts_top1":
        s["y"].zero_()
        s["part"].forward(s["x"], s["y"], s["batch"])
    elif s["kind"] == "experts_top2":
        s["part"].forward(s["x"], s["y"], s["batch"], accumulate=False)
    else:
        if s["cache"].state is not None:
            s["cache"].state.zero_()                    # every request of the step is a new one
        s["part"].forward(s["x"], s["y"], s["batch"], s["cache"], accumulate=False)


def run(s):
    if s["kind"] == "sampling":
        ids, _ = s["sampler"].sample_on_device(s["logits"], s["rows"])
        return ids
    if s["kind"] == "requests":
        engine, seqs = s["engine"], s["seqs"]
        first = engine.step([(i, p, [len(p) - 1]) for i, (p, _) in enumerate(seqs)])
        out = [first.clone()]
        for t in range(s["steps"]):
            out.append(engine.step([(i, [f[t]], [0]) for i, (_, f) in enumerate(seqs)]).clone())
        for i in range(len(seqs)):
            engine.finish(i)
        return out
    if "graph" in s:
        s["graph"].replay()
    else:
        _forward(s)
    out = {"y": s["y"]}
    if s["cache"] is not None:
        out["cache"] = s["cache"].kv if s["cache"].kv is not None else _matrices(s)
    return out


def _matrices(s):
    """The requests' state without what a slot holds besides its matrices (copies of a kernel's own, padding)."""
    state, part = s["cache"].state, s["part"]
    if s["kind"] == "matrix_memory":
        return state[:, :, :part.kd * part.vd]
    return state[:, :part.state_matrices]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "sampling":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n, "flops": 8 * n}
    d = case["width"]
    if kind == "requests":
        mem = 2 * 8 * (d // 16) * d + 3 * d * d
        att = 3 * d * d + 8 * d * d
        head = 32768 * d
        weights = 2 * mem + 2 * att + d * d // 2 + head
        seqs = _sequences(case, 0)
        tokens = sum(len(p) for p, _ in seqs)
        state = 2 * 2 * 8 * (d // 16) * (d // 8) * 4 * case["requests"]
        return {"bytes": (1 + case["steps"]) * (2 * weights + state + 4 * 32768 * case["requests"]),
                "flops": 2 * (weights - head) * (tokens + case["requests"] * case["steps"]) + 2 * head * case["requests"] * (1 + case["steps"])}
    T = case["tokens"]
    io = T * d * (2 + 4)
    if kind == "attention":
        n, m = case["heads"] * 128, case["kv_heads"] * 128
        weights = 2 * d * n + 2 * d * m
        segs = _segments(case)
        seen = sum(sum(p + 1 for p in range(a, a + k)) for a, k in segs)
        keys = sum(a + k for a, k in segs)
        return {"bytes": 2 * weights + io + 2 * 2 * keys * m, "flops": 2 * T * weights + 4 * n * seen}
    if kind == "experts_top1" or kind == "experts_top2":
        E, f = case["experts"], case["inner"]
        top = 1 if kind == "experts_top1" else 2
        per = 3 * d * f
        used = E * (1.0 - (1.0 - top / E) ** T)          # experts that T tokens draw, on average
        shared = per if top == 1 else 0
        return {"bytes": int(2 * (used * per + shared)) + io, "flops": 2 * T * (top * per + shared)}
    H, dk, dv, weights = {"matrix_memory": (8, d // 16, d // 8, 4 * d * d), "delta": (d // 128, 128, 128, 4 * d * d),
                          "state_space": (d // 32, 128, 64, 6 * d * d), "linear_attention": (d // 128, 64, 128, 4 * d * d)}[kind]
    return {"bytes": 2 * weights + io + 4 * case["requests"] * H * dk * dv, "flops": 2 * T * weights + 4 * T * H * dk * dv}


def tolerance(case):
    """Layers round what enters their output projection to bfloat16 (2^-9), the recurrences' matrices stay float32."""
    kind = case["kind"]
    if kind == "sampling":
        return {"rel": 0.0, "differ": 0.01}
    if kind == "requests":
        return {"rel": 0.025}
    return {"rel": 0.01, "max": 0.25}


# ------------------------------------------------------------------ the same in 64 bits
def _f(p):
    return {k: t.double() for k, t in p.items()}


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, w, b):
    """Causal over time, the last tap on the token itself, then silu.  x [T, C], w [C, taps]."""
    n = w.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x], 0)
    y = sum(w[:, j] * padded[j:j + x.shape[0]] for j in range(n))
    return _silu(y if b is None else y + b)


def _memory(x, p, d):
    """The matrix memory on one sequence: (what enters the output projection, the matrices)."""
    H, dk, dv, T = 8, d // 16, d // 8, x.shape[0]
    q, k = (x @ p["q_proj"].T).view(T, H, dk) * dk ** -0.5, (x @ p["k_proj"].T).view(T, H, dk)
    v = (x @ p["v_proj"].T).view(T, H, dv)
    gi = 10.0 * torch.tanh((x @ p["igate_proj"].T + p["igate_bias"]) / 10.0)
    gf = torch.nn.functional.logsigmoid(10.0 * torch.tanh((x @ p["fgate_proj"].T + p["fgate_bias"]) / 10.0))
    S, n, m, out = x.new_zeros(H, dk, dv), x.new_zeros(H, dk), x.new_zeros(H), []
    for t in range(T):
        new = torch.maximum(gf[t] + m, gi[t])
        keep, take = torch.exp(gf[t] + m - new)[:, None], torch.exp(gi[t] - new)[:, None] * k[t]
        m = new
        S = keep[:, :, None] * S + take[:, :, None] * v[t][:, None, :]
        n = keep * n + take
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out.append(torch.einsum("hkv,hk->hv", S, q[t]) / den[:, None])
    o = _rms(torch.stack(out), 1e-5).reshape(T, H * dv) * p["norm"]
    return o * torch.sigmoid(x @ p["gate_proj"].T), S


def _delta(x, p, d):
    H, G, dk, dv, T = d // 128, d // 256, 128, 128, x.shape[0]
    q = _conv(x @ p["q_proj"].T, p["q_conv"], None).view(T, G, dk)
    k = _conv(x @ p["k_proj"].T, p["k_conv"], None).view(T, G, dk)
    v = _conv(x @ p["v_proj"].T, p["v_conv"], None).view(T, H, dv)
    q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5).repeat_interleave(H // G, 1)
    k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    beta = torch.sigmoid(x @ p["beta_proj"].T)
    g = torch.exp(-torch.exp(p["a_log"]) * torch.nn.functional.softplus(x @ p["decay_proj"].T + p["dt_bias"]))
    S, out = x.new_zeros(H, dk, dv), []
    for t in range(T):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]))
    o = (_rms(torch.stack(out), 1e-6) * p["norm"]).reshape(T, H * dv)
    return o * _silu(x @ p["gate_proj"].T), S


def _state_space(x, p, d):
    H, n, N, T = d // 32, 2 * d, 128, x.shape[0]
    z, xbc, a = (x @ p["in_proj"].T).split([n, n + 2 * N, H], 1)
    u, B, C = _conv(xbc, p["conv"], p["conv_bias"]).split([n, N, N], 1)
    u = u.view(T, H, 64)
    dt = torch.nn.functional.softplus(a + p["dt_bias"])
    g = torch.exp(-torch.exp(p["a_log"]) * dt)
    S, out = x.new_zeros(H, 64, N), []                    # (the slot's order: value columns, then keys)
    for t in range(T):
        S = g[t][:, None, None] * S + (dt[t][:, None] * u[t])[:, :, None] * B[t]
        out.append(S @ C[t] + p["skip"][:, None] * u[t])
    return _rms(torch.stack(out).reshape(T, n) * _silu(z), 1e-6) * p["norm"], S


def _linear_attention(x, p, d):
    H, dk, dv, T = d // 128, 64, 128, x.shape[0]
    q, k = (x @ p["q_proj"].T).view(T, H, dk) * dk ** -0.5, (x @ p["k_proj"].T).view(T, H, dk)
    v = (x @ p["v_proj"].T).view(T, H, dv)
    w = torch.sigmoid((x @ p["decay_in"].T) @ p["decay_out"].T + p["decay_bias"]).pow(1 / 16.0).view(T, H, dk)
    S, out = x.new_zeros(H, dv, dk), []
    for t in range(T):
        S = w[t][:, None, :] * S + v[t][:, :, None] * k[t][:, None, :]
        out.append(torch.einsum("hvk,hk->hv", S, q[t]))
    o = (_rms(torch.stack(out), 1e-6) * p["norm"]).reshape(T, H * dv)
    return o * _silu(x @ p["gate_proj"].T), S


def _rotate(x, first, halves):
    """x [T, heads, 128] turned by its position: neighbouring pairs of the whole head, or the halves of its first 64 elements."""
    dims = 64 if halves else 128
    f = 500000.0 ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=torch.float64) / dims)
    a = (torch.arange(first, first + x.shape[0], device=DEV, dtype=torch.float64)[:, None] * f)[:, None, :]
    if halves:
        u, v = x[..., :32], x[..., 32:64]
        return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., 64:]], -1)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)


def _softmax_rows(q, k, v, first):
    """q [T, heads, 128] at the positions from `first` on over k, v [positions, kv heads, 128]."""
    T, group = q.shape[0], q.shape[1] // k.shape[1]
    see = torch.arange(k.shape[0], device=DEV)[None, :] <= torch.arange(first, first + T, device=DEV)[:, None]
    out = [torch.softmax((q[:, h] @ k[:, h // group].T * 128 ** -0.5).masked_fill(~see, -math.inf), -1) @ v[:, h // group]
           for h in range(q.shape[1])]
    return torch.stack(out, 1).reshape(T, -1)


def _exact_attention(case, p, x, kv):
    kv, outs, row, page = kv.double(), [], 0, 0
    for first, n in _segments(case):
        h, pages = x[row:row + n], -(-(first + n) // PAGE)
        heads = lambda name: (h @ p[name].T).view(n, -1, 128)
        q, k, v = _rms(_rotate(heads("q_proj"), first, False), 1e-5), _rms(_rotate(heads("k_proj"), first, False), 1e-5), heads("v_proj")
        at = torch.arange(first, first + n, device=DEV)
        for plane, new in enumerate((k, v)):
            kv[plane, page + at // PAGE, :, at % PAGE] = new
        lay = kv[:, page:page + pages].transpose(2, 3).reshape(2, pages * PAGE, case["kv_heads"], 128)[:, :first + n]
        outs.append(_softmax_rows(q, lay[0], lay[1], first) @ p["o_proj"].T)
        row, page = row + n, page + pages
    return {"y": torch.cat(outs), "cache": kv}


def _exact_experts(case, p, x):
    top = 1 if case["kind"] == "experts_top1" else 2
    logits = x @ p["router"].double().T
    chosen = logits.topk(top, -1).indices
    shares = torch.sigmoid(logits) if top == 1 else torch.softmax(logits, -1)
    y = torch.zeros_like(x)
    if top == 1:
        a = _silu(x @ p["shared_gate_proj"].double().T) * (x @ p["shared_up_proj"].double().T)
        y += a @ p["shared_down_proj"].double().T
    total = shares.gather(1, chosen).sum(1)
    for e in range(case["experts"]):
        rows = (chosen == e).any(1).nonzero()[:, 0]
        if not rows.numel():
            continue
        s, h = shares[rows, e][:, None], x[rows]
        if top == 1:
            gate, up = p["experts_gate_up"][e].double().chunk(2, 0)
            out = (_silu(s * (h @ gate.T)) * (s * (h @ up.T))) @ p["experts_down"][e].double().T
        else:
            out = s / total[rows][:, None] * ((_silu(h @ p["experts_gate"][e].double().T) * (h @ p["experts_up"][e].double().T))
                                              @ p["experts_down"][e].double().T)
        y[rows] += out
    return {"y": y}


def _exact_requests(case, seed):
    p, d = _f(_model_params(case, seed)), case["width"]
    firsts, later = [], [[] for _ in range(case["steps"])]
    for prompt, forced in _sequences(case, seed):
        x = p["embed.weight"][torch.tensor(prompt + forced, device=DEV)]
        kept = None
        for i in range(4):
            w = {k[len(f"layers.{i}."):]: t for k, t in p.items() if k.startswith(f"layers.{i}.")}
            h = _rms(x, 1e-5) * w["mixer_norm.weight"]
            m = {k[6:]: t for k, t in w.items() if k.startswith("mixer.")}
            if i in (0, 3):
                y = _memory(h, m, d)[0] @ m["o_proj"].T
            else:
                heads = lambda s: (h @ m[s + "_proj"].T + m[s + "_bias"]).view(h.shape[0], -1, 128)
                if i == 1:
                    kept = _rotate(heads("k"), 0, True), heads("v")
                o = _softmax_rows(_rotate(heads("q"), 0, True), *kept, 0)
                y = (o * torch.sigmoid(h @ m["out_gate_proj"].T)) @ m["o_proj"].T + m["o_bias"]
            x = x + 0.5 * _rms(y, 1e-5) * w["mixer_out_norm.weight"]
            if i in (1, 2):
                h = _rms(x, 1e-5) * w["ffn_norm.weight"]
                y = torch.nn.functional.gelu(h @ w["ffn.up_proj"].T, approximate="tanh") @ w["ffn.down_proj"].T
                x = x + 0.5 * _rms(y, 1e-5) * w["ffn_out_norm.weight"]
        logits = 0.5 * ((_rms(x[len(prompt) - 1:], 1e-5) * p["final_norm.weight"]) @ p["embed.weight"].T)
        firsts.append(logits[0])
        for t in range(case["steps"]):
            later[t].append(logits[1 + t])
    return [torch.stack(firsts)] + [torch.stack(rows) for rows in later]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sampling":
        return None
    with torch.no_grad():
        if kind == "requests":
            return _exact_requests(case, seed)
        r = _Draws(seed)
        p = _params(case, r)
        x = r.normal(case["tokens"], case["width"]).double()
        if kind.startswith("experts"):
            return _exact_experts(case, p, x)
        if kind == "attention":
            pages = sum(-(-(a + n) // PAGE) for a, n in _segments(case))
            return _exact_attention(case, _f(p), x, r.normal(2, pages, case["kv_heads"], PAGE, 128))
        p = _f(p)
        cell = {"matrix_memory": _memory, "delta": _delta, "state_space": _state_space, "linear_attention": _linear_attention}[kind]
        outs, states, row = [], [], 0
        for _, n in _segments(case):
            o, S = cell(x[row:row + n], p, case["width"])
            outs.append(o @ p["o_proj"].T)
            states.append(S.flatten(1) if kind == "matrix_memory" else S.flatten())
            row += n
        return {"y": torch.cat(outs), "cache": torch.stack(states)}
