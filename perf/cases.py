"""Workloads of the framework as calls of its public entry points: the attention operators of the C ABI (a prompt, one decode
step, fp32 training forward and backward) and the three decoder families (a prompt pass and single-token steps behind it).

listed() names the workloads, draw() takes another one of the same ranges, prepare() holds what a program has in hand before
the call, run() makes one pass, and exact() states the same results in 64-bit torch."""
import ctypes
import math

import numpy as np
import torch

from vesper_b200 import capi, model

THETA = 10000.0
VOCAB, WIDTH, LAYERS, EPS = 32000, 2048, 4, 1e-6
LLAMA = dict(heads=16, kv_heads=4, ff=5632)
LATENT = dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5, rot=dict(base=THETA, dims=64), mask=dict(size=1024))
MAMBA2 = dict(heads=64, vdim=64, state=128, groups=1, conv=4, norm_groups=1)
BIGRAM = dict(buckets=65536, mul_prev=31337, mul_cur=1)
SIGMOID = dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, bias_max=256, v_mix=True, q_temp=dict(coef=0.1, every=1024))
MAMBA1 = dict(inner=4096, state=16, dt_rank=128, conv=4)
MOE = dict(kind="moe", expert=dict(ff=704), router=dict(experts=64, top=6, scale=2.5, groups=dict(count=8, keep=4)), shared=dict(ff=1408))
BIAS_ROWS = 32
NITENEX_FF, ZUDISUN_FF = 8448, 5632


def listed():
    return [
        # a batch of four prompts through one layer's attention, rotation and cache append included
        _prompt("prompt_batch", "bfloat16", 4, 32, 8, 2048, 128),
        # one sequence's next token early in its life: the smallest call, all latency
        _step("step_short", "bfloat16", 1, 16, 4, 300, False, 128),
        # a serving batch with contexts of every length, one token each
        _step("step_ragged", "bfloat16", 32, 32, 8, 8192, True, 128),
        # one sequence with a very long context
        _step("step_long", "bfloat16", 1, 64, 8, 131072, False, 128),
        # a training step's attention of a small model (16 heads of 64, 512 tokens, one sequence), forward and backward
        _train("train_small", 1, 16, 512, 64),
        # the same for two sequences of an odd length and wider heads
        _train("train_odd", 2, 16, 1999, 128),
        # eight prompts through a stack of Llama-style layers
        _model("llama_prompt", "llama", 8, 512, 0),
        # eight sequences generating token by token behind short prompts
        _model("llama_steps", "llama", 8, 96, 16),
        # the hybrid decoder with state-space layers and latent attention: an odd batch of prompts
        _model("nitenex_prompt", "nitenex", 3, 1001, 0),
        # one user's sequence, token by token
        _model("nitenex_steps", "nitenex", 1, 40, 16),
        # the hybrid decoder with selective scans, sigmoid attention and experts: prompts
        _model("zudisun_prompt", "zudisun", 8, 512, 0),
        # a batch of sequences, token by token
        _model("zudisun_steps", "zudisun", 16, 24, 16),
    ]


def draw(rng):
    """One more case: sizes log-uniform over their ranges, so that most are odd."""
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["prompt", "prompt", "step", "step", "train", "llama", "nitenex", "zudisun"])
    while True:
        if kind == "prompt":
            hkv = rng.choice([1, 2, 4, 8])
            c = _prompt("", rng.choice(["bfloat16", "bfloat16", "float16"]), log(1, 8), hkv * rng.choice([1, 2, 4, 8]), hkv, log(16, 8192), rng.choice([64, 128, 128]))
            if rng.random() < 0.3:
                c["start"] = log(16, 8192)                    # the prompt's next portion, behind what the cache holds
            fits = work(c)["flops"] <= work(listed()[0])["flops"] and c["heads"] <= 64
        elif kind == "step":
            hkv = rng.choice([1, 2, 4, 8])
            c = _step("", rng.choice(["bfloat16", "bfloat16", "float16"]), log(1, 64), hkv * rng.choice([1, 2, 4, 8]), hkv, log(64, 131072), rng.random() < 0.5, rng.choice([64, 128, 128]))
            fits = c["B"] * c["kv_heads"] * c["ctx"] <= 32 * 8 * 4608 and c["heads"] <= 64
        elif kind == "train":
            c = _train("", log(1, 4), rng.choice([4, 8, 12, 16]), log(64, 2048), rng.choice([64, 128]))
            fits = work(c)["flops"] <= work(listed()[5])["flops"]
        else:
            c = _model("", kind, log(1, 32), log(16, 2048), rng.choice([0, 4, 12]))
            fits = c["B"] * c["prompt"] <= (512 if c["steps"] else 3500)
        if fits:
            del c["name"]
            return c


def prepare(case, seed):
    return {"prompt": _prepare_prompt, "step": _prepare_step, "train": _prepare_train, "model": _prepare_model}[case["kind"]](case, seed)


def run(state):
    return state["pass"](state)


def exact(case, seed):
    return {"prompt": _exact_prompt, "step": _exact_step, "train": _exact_train, "model": _exact_model}[case["kind"]](case, seed)


def work(case):
    """Bytes and operations a pass cannot do without: inputs read once, outputs written once, products of visible pairs."""
    c = case
    if c["kind"] == "prompt":
        pairs = c["T"] * c["start"] + c["T"] * (c["T"] + 1) // 2
        rows = c["B"] * c["T"]
        moved = 2 * c["D"] * (rows * (2 * c["heads"] + 4 * c["kv_heads"]) + c["B"] * c["kv_heads"] * 2 * c["start"]) + 4 * rows * c["heads"]
        return {"bytes": moved, "flops": 4 * c["D"] * c["B"] * c["heads"] * pairs}
    if c["kind"] == "step":
        keys = c["B"] * c["ctx"] * (0.5625 if c["ragged"] else 1)          # ragged lengths are uniform from an eighth of ctx to ctx
        return {"bytes": 4 * c["D"] * (keys * c["kv_heads"] + c["B"] * (c["heads"] + 2 * c["kv_heads"])), "flops": 4 * c["D"] * c["heads"] * keys}
    if c["kind"] == "train":
        rows = c["B"] * c["H"] * c["N"]
        # forward: q, k, v in, output and row sums out; backward: those and the output's gradient in, three gradients out
        return {"bytes": 4 * rows * (12 * c["D"] + 2), "flops": 14 * c["D"] * rows * (c["N"] + 1) // 2}
    return _model_work(c)


def tolerance(case):
    if case["kind"] == "train":
        return {"rel": 1e-5}
    if case["kind"] in ("prompt", "step"):
        return {"rel": 1e-2 if case["dtype"] == "bfloat16" else 2e-3}
    return {"rel": 3e-2, "max": 0.6}


# ---- attention operators ------------------------------------------------------------------------

def _prompt(name, dtype, B, heads, kv_heads, T, D):
    return dict(name=name, kind="prompt", dtype=dtype, B=B, heads=heads, kv_heads=kv_heads, T=T, D=D, start=0)


def _step(name, dtype, B, heads, kv_heads, ctx, ragged, D):
    return dict(name=name, kind="step", dtype=dtype, B=B, heads=heads, kv_heads=kv_heads, ctx=ctx, ragged=ragged, D=D)


def _train(name, B, H, N, D):
    return dict(name=name, kind="train", B=B, H=H, N=N, D=D)


def _random(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _prompt_inputs(c, seed):
    g, dt = _random(seed), getattr(torch, c["dtype"])
    B, Hq, Hkv, T, D = (c[k] for k in ("B", "heads", "kv_heads", "T", "D"))
    s = dict(q=_randn(g, B, Hq, T, D, dtype=dt, scale=0.5), k=_randn(g, B, Hkv, T, D, dtype=dt, scale=0.5), v=_randn(g, B, Hkv, T, D, dtype=dt, scale=0.5))
    cap = max(c["start"] + T, 4096 if T <= 4096 else 8192)
    for name in ("k_cache", "v_cache"):
        s[name] = torch.zeros(B, Hkv, cap, D, dtype=dt, device="cuda")
        if c["start"]:
            s[name][:, :, :c["start"]] = _randn(g, B, Hkv, c["start"], D, dtype=dt, scale=0.5)
    return s


def _prepare_prompt(c, seed):
    s = _prompt_inputs(c, seed)
    s["o"] = torch.empty_like(s["q"])
    s["lse"] = torch.empty(c["B"], c["heads"], c["T"], device="cuda")
    lib = capi.load()
    args = capi.prefill_args(s["q"], s["k"], s["v"], s["o"], s["lse"], scale=c["D"] ** -0.5, causal=True, start_pos=c["start"], theta=THETA,
                             k_cache=s["k_cache"], v_cache=s["v_cache"])
    s["workspace"] = torch.empty(max(1, lib.vb200_prefill_workspace_bytes(ctypes.byref(args))), dtype=torch.uint8, device="cuda")
    args.workspace, args.workspace_bytes = s["workspace"].data_ptr(), s["workspace"].numel()
    s["args"], s["call"], s["pass"] = args, lib.vb200_prefill_fwd, _run_prompt
    return s


def _run_prompt(s):
    capi.check(s["call"](ctypes.byref(s["args"])))
    return {k: s[k] for k in ("o", "lse", "k_cache", "v_cache")}


def _rotate(x, positions):
    """Adjacent dimensions (2i, 2i + 1) turned by position * theta^(-2i/D); positions broadcast over x's rows."""
    D = x.shape[-1]
    f = (THETA ** (-torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)).float().double()
    a = positions[..., None].double() * f
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], dim=-1).flatten(-2)


def _exact_prompt(c, seed):
    s = _prompt_inputs(c, seed)
    T, start, group = c["T"], c["start"], c["heads"] // c["kv_heads"]
    at = torch.arange(start, start + T, device="cuda")
    kc, vc = s["k_cache"].double(), s["v_cache"].double()
    kc[:, :, start:start + T] = _rotate(s["k"].double(), at)
    vc[:, :, start:start + T] = s["v"].double()
    o = torch.empty(s["q"].shape, dtype=torch.float64, device="cuda")
    lse = torch.empty(s["q"].shape[:3], dtype=torch.float64, device="cuda")
    for b in range(c["B"]):
        for h in range(c["heads"]):
            k, v = kc[b, h // group, :start + T], vc[b, h // group, :start + T]
            for r in range(0, T, 2048):
                q = _rotate(s["q"][b, h, r:r + 2048].double(), at[r:r + 2048])
                w = (q @ k.T) * c["D"] ** -0.5
                w.masked_fill_(torch.arange(start + T, device="cuda")[None] > at[r:r + 2048, None], -math.inf)
                lse[b, h, r:r + 2048] = torch.logsumexp(w, -1)
                o[b, h, r:r + 2048] = torch.softmax(w, -1) @ v
    return {"o": o, "lse": lse, "k_cache": kc, "v_cache": vc}


def _step_inputs(c, seed):
    g, dt = _random(seed), getattr(torch, c["dtype"])
    B, Hq, Hkv, D, ctx = (c[k] for k in ("B", "heads", "kv_heads", "D", "ctx"))
    cap = (ctx + 64) // 64 * 64
    s = dict(q=_randn(g, B, Hq, 1, D, dtype=dt), k=_randn(g, B, Hkv, 1, D, dtype=dt), v=_randn(g, B, Hkv, 1, D, dtype=dt),
             k_cache=torch.randn(B, Hkv, cap, D, generator=g, device="cuda", dtype=dt), v_cache=torch.randn(B, Hkv, cap, D, generator=g, device="cuda", dtype=dt))
    lens = np.random.default_rng(seed).integers(max(1, ctx // 8), ctx + 1, size=B) if c["ragged"] else np.full(B, ctx)
    s["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
    s["longest"] = int(lens.max())
    return s


def _prepare_step(c, seed):
    s = _step_inputs(c, seed)
    s["o"] = torch.empty_like(s["q"])
    lib = capi.load()
    where = dict(seq_lens=s["lens"]) if c["ragged"] else dict(uniform_len=c["ctx"])
    args = capi.decode_args(s["q"], s["o"], s["k_cache"], s["v_cache"], scale=c["D"] ** -0.5, k_new=s["k"], v_new=s["v"], theta=THETA, max_len=s["longest"] + 1, **where)
    s["workspace"] = torch.empty(max(1, lib.vb200_decode_workspace_bytes(ctypes.byref(args))), dtype=torch.uint8, device="cuda")
    args.workspace, args.workspace_bytes = s["workspace"].data_ptr(), s["workspace"].numel()
    s["args"], s["call"], s["pass"] = args, lib.vb200_decode_fwd, _run_step
    return s


def _run_step(s):
    capi.check(s["call"](ctypes.byref(s["args"])))
    return {k: s[k] for k in ("o", "k_cache", "v_cache")}


def _exact_step(c, seed):
    s = _step_inputs(c, seed)
    group = c["heads"] // c["kv_heads"]
    o = torch.empty(s["q"].shape, dtype=torch.float64, device="cuda")
    for b, n in enumerate(s["lens"].tolist()):
        at = torch.tensor([n], device="cuda")
        for h in range(c["kv_heads"]):
            q = _rotate(s["q"][b, h * group:(h + 1) * group].double(), at)[:, 0]
            k = torch.cat([s["k_cache"][b, h, :n].double(), _rotate(s["k"][b, h].double(), at)])
            v = torch.cat([s["v_cache"][b, h, :n].double(), s["v"][b, h].double()])
            o[b, h * group:(h + 1) * group, 0] = torch.softmax((q @ k.T) * c["D"] ** -0.5, -1) @ v
    return {"o": o, "k_cache": None, "v_cache": None}


def _train_inputs(c, seed):
    g = _random(seed)
    return {k: _randn(g, c["B"], c["H"], c["N"], c["D"]) for k in ("q", "k", "v", "d_out")}


def _prepare_train(c, seed):
    s = _train_inputs(c, seed)
    s["o"], s["scale"] = torch.empty_like(s["q"]), c["D"] ** -0.5
    s["lse"] = torch.empty(c["B"], c["H"], c["N"], device="cuda")
    s["pass"] = _run_train
    return s


def _run_train(s):
    capi.prefill(s["q"], s["k"], s["v"], s["o"], s["lse"], scale=s["scale"], causal=True)
    dq, dk, dv = capi.attention_bwd(s["d_out"], s["q"], s["k"], s["v"], s["o"], s["lse"], scale=s["scale"], causal=True)
    return {"o": s["o"], "lse": s["lse"], "dq": dq, "dk": dk, "dv": dv}


def _exact_train(c, seed):
    s = {k: v.double() for k, v in _train_inputs(c, seed).items()}
    out = {k: torch.empty_like(s["q"]) for k in ("o", "dq", "dk", "dv")}
    out["lse"] = torch.empty(s["q"].shape[:3], dtype=torch.float64, device="cuda")
    hidden = torch.ones(c["N"], c["N"], dtype=torch.bool, device="cuda").triu(1)
    scale = c["D"] ** -0.5
    for b in range(c["B"]):
        for h in range(c["H"]):
            q, k, v, g = (s[n][b, h] for n in ("q", "k", "v", "d_out"))
            w = (q @ k.T * scale).masked_fill_(hidden, -math.inf)
            out["lse"][b, h] = torch.logsumexp(w, -1)
            p = torch.softmax(w, -1)
            out["o"][b, h] = p @ v
            ds = p * (g @ v.T - (g * out["o"][b, h]).sum(-1, keepdim=True)) * scale
            out["dq"][b, h], out["dk"][b, h], out["dv"][b, h] = ds @ k, ds.T @ q, p.T @ g
    return out


# ---- decoders -----------------------------------------------------------------------------------

def _model(name, family, B, prompt, steps):
    return dict(name=name, kind="model", family=family, B=B, prompt=prompt, steps=steps)


def _config(family):
    """One period of the family's layers: four attention layers, or three state-space layers and one of attention."""
    if family == "nitenex":
        layers = [dict(type="latent_attention" if i % 4 == 3 else "mamba2", mixer=LATENT if i % 4 == 3 else MAMBA2, mlp=dict(kind="dense", ff=NITENEX_FF)) for i in range(LAYERS)]
        return dict(architecture="Nitenex", vocab=VOCAB, width=WIDTH, norm=dict(eps=EPS), layers=layers, embedding=dict(bigram=BIGRAM))
    layers = [dict(type="attention" if i % 4 == 3 else "mamba1", mixer=SIGMOID if i % 4 == 3 else MAMBA1, mlp=MOE if i % 4 == 3 else dict(kind="dense", ff=ZUDISUN_FF))
              for i in range(LAYERS)]
    return dict(architecture="Zudisun", vocab=VOCAB, width=WIDTH, norm=dict(eps=EPS), layers=layers)


def _new_model(c):
    longest = c["prompt"] + c["steps"]
    if c["family"] == "llama":
        return model.TransformerLM(VOCAB, WIDTH, LAYERS, LLAMA["heads"], LLAMA["kv_heads"], LLAMA["ff"], longest)
    return model.model_from_config(_config(c["family"]), "bfloat16", max_seq_len=longest, max_sequences=c["B"])


def _weights(shapes, seed):
    """(name, values) of every parameter, all of them numbers that bf16 holds: matrices 0.02 N(0, 1) cut from one pool, norms and
    gains around one, step-size biases around -3, decays from 1 to 16.  The norms that end the experts' layers have a tenth of that
    gain: a token whose router is undecided between two experts may take either, and then moves a little and not a lot."""
    g = torch.Generator().manual_seed(seed)
    pool = (torch.randn(1 << 24, generator=g) * 0.02).bfloat16().float()
    for i, (name, shape) in enumerate(sorted(shapes.items())):
        shape = tuple(BIAS_ROWS if d < 0 else d for d in shape)
        n, at = math.prod(shape), 977 * i % 65536
        x = pool[at:at + n] if at + n <= pool.numel() else pool.repeat(-(-(at + n) // pool.numel()))[at:at + n]
        x = x.view(shape)
        last = name.rsplit(".", 1)[-1]
        if len(shape) == 1 and (last in ("norm", "norm1", "norm2", "D") or "norm.weight" in name):
            x = (x * 5 + 1) * (0.1 if "l%d.norm2" % (LAYERS - 1) == name and any(".router" in n for n in shapes) else 1.0)
        elif last == "dt_bias" or name.endswith("dt.b"):
            x = x * 25 - 3
        elif last == "A_log":
            x = x + torch.linspace(1, 16, shape[-1]).log()
        elif last == "pb":
            x = x - 5
        elif last == "talk":
            x = x + torch.eye(shape[0])
        elif last == "conv":
            x = x * 25
        yield name, x.bfloat16().float()


def _ids(c, seed):
    return np.random.default_rng(seed).integers(0, VOCAB, size=(c["B"], c["prompt"] + c["steps"])).astype(np.int32)


def _shapes(m):
    return model.param_shapes(VOCAB, WIDTH, LAYERS, LLAMA["heads"], LLAMA["kv_heads"], LLAMA["ff"]) if isinstance(m, model.TransformerLM) else m.param_shapes()


def _prepare_model(c, seed):
    m = _new_model(c)
    for name, x in _weights(_shapes(m), seed):
        m.set_param(name, x.numpy())
    m.init_cache(c["B"])
    return {"model": m, "ids": _ids(c, seed), "prompt": c["prompt"], "pass": _run_model}


def _run_model(s):
    """The prompts, then the given tokens one at a time: the next token's logits after each call."""
    m, ids, P = s["model"], s["ids"], s["prompt"]
    out = [m.forward_with_cache(ids[:, :P], 0, last_only=True)]
    for t in range(P, ids.shape[1]):
        out.append(m.forward_with_cache(ids[:, t:t + 1], t, last_only=True))
    return out


def _model_work(c):
    B, P, S = c["B"], c["prompt"], c["steps"]
    d = WIDTH
    if c["family"] == "llama":
        hd = d // LLAMA["heads"]
        dense = LAYERS * (d * hd * (2 * LLAMA["heads"] + 2 * LLAMA["kv_heads"]) + 3 * d * LLAMA["ff"])
        per_pair, key_bytes, experts = LAYERS * 4 * d, LAYERS * 4 * LLAMA["kv_heads"] * hd, 0
        token_flops, state_bytes = 2 * dense, 0
    elif c["family"] == "nitenex":
        l, m = LATENT, MAMBA2
        inner = m["heads"] * m["vdim"]
        dense = 4 * 2 * d * NITENEX_FF + 3 * d * (3 * inner + 2 * m["state"] + m["heads"]) + d * (l["heads"] * (l["dim"] + l["rot_dim"]) + l["kv_rank"] + l["rot_dim"]) \
            + l["heads"] * l["kv_rank"] * (l["dim"] + l["vdim"]) + l["heads"] * l["vdim"] * d
        per_pair, key_bytes, experts = 2 * l["heads"] * (l["dim"] + l["rot_dim"] + l["vdim"]), 2 * (l["kv_rank"] + l["rot_dim"]), 0
        token_flops, state_bytes = 2 * dense + 3 * 5 * inner * m["state"], 3 * 4 * inner * m["state"]
    else:
        a, m, r = SIGMOID, MAMBA1, MOE["router"]
        dense = 3 * (3 * d * ZUDISUN_FF + 3 * d * m["inner"] + m["inner"] * (2 * m["dt_rank"] + 2 * m["state"])) \
            + d * (a["heads"] * (a["dim"] + 1 + a["vdim"]) + a["kv_heads"] * (a["dim"] + a["vdim"])) + 3 * d * MOE["shared"]["ff"] + d * r["experts"]
        per_pair, key_bytes = 2 * a["heads"] * (a["dim"] + a["vdim"] + a["heads"]), 2 * a["kv_heads"] * (a["dim"] + a["vdim"])
        experts = 3 * d * MOE["expert"]["ff"]
        token_flops, state_bytes = 2 * (dense + r["top"] * experts) + 3 * 6 * m["inner"] * m["state"], 3 * 4 * m["inner"] * m["state"]
    hit = lambda tokens: 64 * (1 - (1 - 6 / 64) ** tokens) if experts else 0          # experts that this many tokens choose, on average
    head = d * VOCAB
    flops = B * (P + S) * token_flops + 2 * B * (1 + S) * head + B * per_pair * sum(min(t + 1, 1024 if c["family"] == "nitenex" else t + 1) for t in range(P + S))
    moved = (1 + S) * 2 * (dense + head) + 2 * experts * (hit(B * P) + S * hit(B)) + (1 + S) * B * 4 * VOCAB
    moved += B * sum(key_bytes * (P + s + 1) for s in range(S)) + B * P * key_bytes + B * (1 + 2 * S) * state_bytes
    return {"bytes": moved, "flops": flops}


class _Exact:
    """The decoders' equations over whole sequences in 64 bits, every token's logits from one pass."""

    def __init__(self, c, seed):
        shapes = model.param_shapes(VOCAB, WIDTH, LAYERS, LLAMA["heads"], LLAMA["kv_heads"], LLAMA["ff"]) if c["family"] == "llama" else None
        if shapes is None:
            m = _new_model(c)
            shapes = m.param_shapes()
            m.close()
        self.w = {n: x.to("cuda") for n, x in _weights(shapes, seed)}
        self.c, self.ids = c, torch.from_numpy(_ids(c, seed)).long().cuda()
        self.T = self.ids.shape[1]

    def lin(self, x, name):
        return x @ self.w[name].double().T + (self.w[name + ".b"].double() if name + ".b" in self.w else 0.0)

    def vec(self, name):
        return self.w[name].double()

    @staticmethod
    def rms(x):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)

    def heads(self, x, n):
        return x.unflatten(-1, (n, -1)).transpose(1, 2)

    def logits(self):
        at = range(self.c["prompt"] - 1, self.T)
        if self.c["family"] == "llama":
            h, head, norm = self.llama(), "output.weight", "norm.weight"
        else:
            h, head, norm = getattr(self, self.c["family"])(), "embed" if self.c["family"] == "nitenex" else "head", "final.norm"
        h = self.rms(h[:, list(at)]) * self.vec(norm)
        y = h @ self.w[head].double().T
        return [y[:, i:i + 1].clone() for i in range(len(at))]

    def llama(self):
        F = torch.nn.functional
        H, G, at = LLAMA["heads"], LLAMA["kv_heads"], torch.arange(self.T, device="cuda")
        D = WIDTH // H
        hidden = at[None] > at[:, None]
        h = self.w["tok_embeddings.weight"][self.ids].double()
        for i in range(LAYERS):
            p = "layers.%d." % i
            x = self.lin(self.rms(h) * self.vec(p + "attention_norm.weight"), p + "attention.wqkv.weight")
            q, k, v = self.heads(x[..., :H * D], H), self.heads(x[..., H * D:(H + G) * D], G), self.heads(x[..., (H + G) * D:], G)
            q, k = _rotate(q, at), _rotate(k, at)
            o = torch.empty_like(q)
            for j in range(H):
                w = (q[:, j] @ k[:, j * G // H].transpose(1, 2) * D ** -0.5).masked_fill_(hidden, -math.inf)
                o[:, j] = torch.softmax(w, -1) @ v[:, j * G // H]
            h = h + self.lin(o.transpose(1, 2).flatten(2), p + "attention.wo.weight")
            x = self.rms(h) * self.vec(p + "ffn_norm.weight")
            h = h + self.lin(F.silu(self.lin(x, p + "feed_forward.gate_proj.weight")) * self.lin(x, p + "feed_forward.up_proj.weight"), p + "feed_forward.down_proj.weight")
        return h

    def conv(self, x, p):
        w = self.vec(p + "conv")
        taps = w.shape[1]
        full = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
        return torch.nn.functional.silu(sum(full[:, t:t + self.T] * w[:, t] for t in range(taps)) + self.vec(p + "conv.b"))

    def mamba2(self, x, p):
        m, F = MAMBA2, torch.nn.functional
        H, P, N = m["heads"], m["vdim"], m["state"]
        inner = H * P
        u = self.lin(x, p + "in")
        xbc = self.conv(u[..., inner:2 * inner + 2 * N], p)
        dt = F.softplus(u[..., 2 * inner + 2 * N:] + self.vec(p + "dt_bias"))
        xs, b, c = xbc[..., :inner].unflatten(-1, (H, P)), xbc[..., inner:inner + N], xbc[..., inner + N:]
        decay, y = torch.exp(-torch.exp(self.vec(p + "A_log")) * dt), torch.empty_like(xs)
        S = torch.zeros(x.shape[0], H, P, N, dtype=torch.float64, device="cuda")
        for t in range(self.T):
            S.mul_(decay[:, t, :, None, None]).add_((dt[:, t, :, None] * xs[:, t])[..., None] * b[:, t, None, None])
            y[:, t] = (S @ c[:, t, None, :, None])[..., 0]
        y = (y + self.vec(p + "D")[:, None] * xs).flatten(2) * F.silu(u[..., :inner])
        return self.lin(self.rms(y) * self.vec(p + "norm"), p + "o")

    def latent(self, x, p):
        m, at = LATENT, torch.arange(self.T, device="cuda")
        H, d, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        f = THETA ** (-torch.arange(0, r, 2, dtype=torch.float64, device="cuda") / r)
        ang = at[:, None].double() * f

        def turn(z):                                    # dimension i with i + r/2
            u, v = z[..., :r // 2], z[..., r // 2:]
            return torch.cat([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()], -1)
        q = self.heads(self.lin(x, p + "q"), H)
        ckv = self.lin(x, p + "dkv")
        lat, kr = self.rms(ckv[..., :rank]) * self.vec(p + "dkv.norm"), turn(ckv[..., rank:])
        qr, k, v = turn(q[..., d:]), self.heads(self.lin(lat, p + "uk"), H), self.heads(self.lin(lat, p + "uv"), H)
        n = at[:, None] - at[None]
        hidden = (n < 0) | (n >= m["mask"]["size"])
        o = torch.empty(q.shape[0], H, self.T, m["vdim"], dtype=torch.float64, device="cuda")
        for j in range(H):
            s = (q[:, j, :, :d] @ k[:, j].transpose(1, 2) + qr[:, j] @ kr.transpose(1, 2)) * m["scale"]
            s = torch.cat([s.masked_fill_(hidden, -math.inf), self.vec(p + "sink")[j].expand(s.shape[0], self.T, 1)], -1)
            o[:, j] = torch.softmax(s, -1)[..., :-1] @ v[:, j]
        return self.lin(o.transpose(1, 2).flatten(2), p + "o")

    def nitenex(self):
        prev = torch.nn.functional.pad(self.ids[:, :-1], (1, 0))
        rows = (prev * BIGRAM["mul_prev"] + self.ids * BIGRAM["mul_cur"]) % BIGRAM["buckets"]
        rows[:, 0] = BIGRAM["buckets"]
        h = self.w["embed"][self.ids].double() + self.w["bigram"][rows].double()
        for i in range(LAYERS):
            p = "l%d." % i
            x = self.rms(h) * self.vec(p + "norm1")
            h = h + (self.latent(x, p + "mix.") if i % 4 == 3 else self.mamba2(x, p + "mix."))
            x = self.rms(h) * self.vec(p + "norm2")
            h = h + self.lin(torch.relu(self.lin(x, p + "mlp.up")).square(), p + "mlp.down")
        return h

    def mamba1(self, x, p):
        m, F = MAMBA1, torch.nn.functional
        inner, N, R = m["inner"], m["state"], m["dt_rank"]
        u = self.lin(x, p + "in")
        c = self.conv(u[..., :inner], p)
        d = self.lin(c, p + "x")
        dt = F.softplus(d[..., :R] @ self.vec(p + "dt").T + self.vec(p + "dt.b"))
        A, y = -torch.exp(self.vec(p + "A_log")), torch.empty_like(c)
        S = torch.zeros(x.shape[0], inner, N, dtype=torch.float64, device="cuda")
        for t in range(self.T):
            S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * c[:, t])[..., None] * d[:, t, None, R:R + N]
            y[:, t] = (S @ d[:, t, R + N:, None])[..., 0]
        return self.lin((y + self.vec(p + "D") * c) * F.silu(u[..., inner:]), p + "o")

    def sigmoid(self, x, p):
        m, at = SIGMOID, torch.arange(self.T, device="cuda")
        H, G = m["heads"], m["kv_heads"]
        q, k, v = self.rms(self.heads(self.lin(x, p + "q"), H)), self.rms(self.heads(self.lin(x, p + "k"), G)), self.heads(self.lin(x, p + "v"), G)
        q = q * (1 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]).double() + 1))[:, None]
        half, reach = BIAS_ROWS // 2, m["bias_max"]
        far = [n if n < half else min(BIAS_ROWS - 1, half + int(math.floor(math.log(n / half) / math.log(reach / half) * (BIAS_ROWS - half) + 1e-9))) for n in range(self.T)]
        rel = self.vec(p + "rel")[torch.tensor(far, device="cuda")]                       # [distance, head]
        n = at[:, None] - at[None]
        bias = rel[n.clamp(min=0)].permute(2, 0, 1)
        o = torch.empty(q.shape[0], H, self.T, m["vdim"], dtype=torch.float64, device="cuda")
        for b in range(q.shape[0]):
            s = q[b] @ k[b].repeat_interleave(H // G, 0).transpose(1, 2) * m["scale"] + bias
            s = torch.sigmoid(torch.einsum("gh,hqk->gqk", self.vec(p + "talk"), s) + self.vec(p + "pb")[:, None, None]).masked_fill_(n < 0, 0.0)
            o[b] = s @ v[b].repeat_interleave(H // G, 0)
        o = o * torch.sigmoid(self.heads(self.lin(x, p + "g"), H))
        return self.lin(o.transpose(1, 2).flatten(2), p + "o")

    def gated(self, x, p, act):
        return self.lin(act(self.lin(x, p + ".gate")) * self.lin(x, p + ".up"), p + ".down")

    def experts(self, x, p):
        r, F = MOE["router"], torch.nn.functional
        E, n, keep = r["experts"], r["groups"]["count"], r["groups"]["keep"]
        s = torch.sigmoid(x @ self.vec(p + ".router").T)
        choice = s + self.vec(p + ".correction")
        score = choice.unflatten(-1, (n, E // n)).topk(2, -1).values.sum(-1)
        kept = torch.zeros_like(score).scatter_(-1, score.topk(keep, -1).indices, 1.0).repeat_interleave(E // n, -1)
        ids = choice.masked_fill(kept == 0, -math.inf).topk(r["top"], -1).indices
        w = s.gather(-1, ids)
        w = w / (w.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = self.gated(x, p + ".shared", F.silu)
        for e in range(E):
            b, t, j = (ids == e).nonzero(as_tuple=True)
            if b.numel():
                out[b, t] += w[b, t, j, None] * self.gated(x[b, t], "%s.e%d" % (p, e), F.silu)
        return out

    def zudisun(self):
        h = self.w["embed"][self.ids].double()
        for i in range(LAYERS):
            p = "l%d." % i
            h = h + self.rms(self.sigmoid(h, p + "mix.") if i % 4 == 3 else self.mamba1(h, p + "mix.")) * self.vec(p + "norm1")
            y = self.experts(h, p + "mlp") if i % 4 == 3 else self.gated(h, p + "mlp", torch.relu)
            h = h + self.rms(y) * self.vec(p + "norm2")
        return h


def _exact_model(c, seed):
    return _Exact(c, seed).logits()
