"""What this framework is asked to do in earnest, as cases that can be timed and checked.

Five kinds of work, each through the package's public entry points:

* ``linear``     the isolated int4 Linear of GPT-2's shapes, one call per (K, N), device buffers in and out;
* ``prompt_attention`` / ``step_attention``  causal attention of new rows, and one query row per sequence
  against a filled fp16 cache;
* ``gpt2``       greedy generation: a decode session's prompt pass and its steps, tokens and last logits out;
* ``hybrid``     the same of a hybrid decoder (gated delta rule and latent attention layers);
* ``serve``      requests of unequal length through the serving step: one step of prompts, then single tokens.

The models' weights are fixed (a program keeps its model while the requests change); prompts, activations and
caches come from the seed.  int4 models are given weights that lie on their quantisation grid, so that the plain
64-bit statement below multiplies the same numbers, and every model's output matrix ties each token to one other
token, so that a greedy pick wins by several standard deviations as it does in a trained model: picks do not hang
on the rounding of near-ties, and every output can be compared.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "async-gpu_b200"))
import b200nn  # noqa: E402
from b200nn import ops, synth  # noqa: E402

GROUP = 128
SHAPES = {"small": ((768, 3072), (3072, 768), (768, 2304), (768, 50257)),
          "xl": ((1600, 4800), (1600, 1600), (1600, 6400), (6400, 1600))}
MODELS = {"small-f32": ("small", False), "small-int4": ("small", True), "xl-int4": ("xl", True)}
DISTINCT_LAYERS = 4  # the layers of a GPT-2 model repeat these (each holds a copy of its own on the device)
HYBRIDS = {"vivezen": (1024, 8, 32000, 8, 4, 128, 64, 256, 512, 512, 2816)}
ZUFILORN = dict(width=1024, layers=8, vocab=32000, heads=8, kv_heads=4, dim=64, vdim=128, ff=2816, positions=2048, streams=2)
ZUFILORN_RANK = 128


def listed():
    return [
        # the isolated Linear of the benchmark's second configuration: one token, a few, a batch
        {"name": "linear-1", "kind": "linear", "shapes": "small", "rows": 1},
        {"name": "linear-8", "kind": "linear", "shapes": "small", "rows": 8},
        {"name": "linear-64", "kind": "linear", "shapes": "small", "rows": 64},
        # isolated attention of the fourth configuration: a prompt of 1024, and a step over 1024 cached positions
        {"name": "prompt-attention-8x1024", "kind": "prompt_attention", "batch": 8, "heads": 12, "seq": 1024, "past": 0},
        {"name": "step-attention-64x1024", "kind": "step_attention", "batch": 64, "heads": 12, "ctx": 1024},
        # the first configuration: one user, the unquantised model, 64 tokens after a prompt of 64
        {"name": "small-f32-1x64+64", "kind": "gpt2", "model": "small-f32", "batch": 1, "prompt": 64, "new": 64},
        # the third: a batch of 32 with long prompts and long answers
        {"name": "small-int4-32x512+256", "kind": "gpt2", "model": "small-int4", "batch": 32, "prompt": 512, "new": 256},
        # one user of the large model, a prompt of no round size
        {"name": "xl-int4-1x77+60", "kind": "gpt2", "model": "xl-int4", "batch": 1, "prompt": 77, "new": 60},
        # the fifth configuration, as one of eight GPUs serves its share, and as one GPU serves all
        {"name": "xl-int4-32x128+128", "kind": "gpt2", "model": "xl-int4", "batch": 32, "prompt": 128, "new": 128},
        {"name": "xl-int4-256x128+128", "kind": "gpt2", "model": "xl-int4", "batch": 256, "prompt": 128, "new": 128},
        # the hybrid decoder's benchmark: prompts of 1024, 32 tokens each
        {"name": "vivezen-64x1024+32", "kind": "hybrid", "model": "vivezen", "batch": 64, "prompt": 1024, "new": 32},
        # a server's step: 24 requests of unequal prompts up to 1000 tokens, then eight tokens each
        {"name": "zufilorn-serve-24x1000+8", "kind": "serve", "model": "zufilorn", "requests": 24, "longest": 1000, "new": 8},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "prompt_attention", "step_attention", "gpt2", "gpt2", "gpt2", "hybrid", "serve"])
    if kind == "linear":
        return {"kind": kind, "shapes": rng.choice(["small", "xl"]), "rows": _log(rng, 1, 300)}
    if kind == "prompt_attention":
        seq = _log(rng, 3, 1000)
        return {"kind": kind, "batch": _log(rng, 1, 16), "heads": rng.choice([12, 25]), "seq": seq, "past": rng.choice([0, 0, rng.randrange(0, 1024 - seq)])}
    if kind == "step_attention":
        return {"kind": kind, "batch": _log(rng, 1, 128), "heads": rng.choice([12, 25]), "ctx": _log(rng, 17, 1024)}
    if kind == "gpt2":
        model = rng.choice(sorted(MODELS))
        return {"kind": kind, "model": model, "batch": _log(rng, 1, 128 if model == "xl-int4" else 64), "prompt": _log(rng, 5, 400),
                "new": _log(rng, 4, 100)}
    if kind == "hybrid":
        return {"kind": kind, "model": "vivezen", "batch": _log(rng, 1, 48), "prompt": _log(rng, 5, 1100), "new": _log(rng, 2, 40)}
    return {"kind": kind, "model": "zufilorn", "requests": _log(rng, 1, 32), "longest": _log(rng, 10, 1100), "new": _log(rng, 1, 16)}


# ---- weights (fixed) -------------------------------------------------------------------------------
_kept = {}


def _once(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _registry():
    return _once("registry", b200nn.KernelRegistry.init_default)


def _gen(*seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.SeedSequence([int(s) for s in seed]).generate_state(1)[0]))
    return g


def _normal(g, *shape, std=1.0):
    return torch.randn(shape, generator=g, device="cuda") * std


def _on_grid(w):
    """w [K, N] moved to its int4 grid: groups of 128 along K, nibbles of -7..7 around scales that fp16 holds, the
    largest nibble of a group 7."""
    K, N = w.shape
    pad = (-K) % GROUP
    g = torch.nn.functional.pad(w, (0, 0, 0, pad)).reshape(-1, GROUP, N)
    top = g.abs().amax(1, keepdim=True)
    s = (top / 7.0).half().float()
    q = torch.where(g.abs() == top, torch.sign(g) * 7.0, torch.clamp(torch.round(g / s), -7, 7))
    return (q * s).reshape(-1, N)[:K].contiguous()


def _gpt2_tensors(model):
    """(config, tensors on the host by checkpoint name, distinct layers only)."""
    size, int4 = MODELS[model]
    cfg = getattr(b200nn.Gpt2Config, size)()
    d, V, P = cfg.n_embd, cfg.vocab_size, cfg.n_positions
    g = _gen(17, d, int(int4))
    grid = _on_grid if int4 else (lambda w: w)
    half = grid(_normal(g, d, (V + 1) // 2, std=0.5)).T
    sign = torch.where(torch.rand(d, generator=g, device="cuda") < 0.5, -1.0, 1.0)
    wte = torch.stack([half, half * sign], 1).reshape(-1, d)[:V]  # token 2i + 1 is token 2i with some signs turned
    out = {"wte": wte, "wpe": _normal(g, P, d, std=0.02), "ln_f.weight": sign, "ln_f.bias": torch.zeros(d, device="cuda")}
    for i in range(DISTINCT_LAYERS):
        p = f"h.{i}."
        for n in ("ln_1", "ln_2"):
            out[p + n + ".weight"] = 1.0 + _normal(g, d, std=0.1)
            out[p + n + ".bias"] = _normal(g, d, std=0.1)
        for n, k, m in (("attn.c_attn", d, 3 * d), ("attn.c_proj", d, d), ("mlp.c_fc", d, 4 * d), ("mlp.c_proj", 4 * d, d)):
            std = 0.02 if m != d else 0.02 * (2 * cfg.n_layer) ** -0.5  # what adds to the residual stream shrinks with the depth
            out[p + n + ".weight"] = grid(_normal(g, k, m, std=std))
            out[p + n + ".bias"] = _normal(g, m, std=0.02)
    return cfg, {n: t.cpu().numpy() for n, t in out.items()}


def _gpt2_model(model):
    def make():
        cfg, w = _gpt2_tensors(model)
        full = {n: a for n, a in w.items() if not n.startswith("h.")}
        for i in range(cfg.n_layer):
            src = f"h.{i % DISTINCT_LAYERS}."
            full.update({f"h.{i}." + n[len(src):]: a for n, a in w.items() if n.startswith(src)})
        if MODELS[model][1]:
            return b200nn.Int4Gpt2Model(full, cfg, _registry(), flags=b200nn.QUANT_LM_HEAD, group_size=GROUP)
        return b200nn.Gpt2Model(full, cfg, _registry())
    return _once(model, make)


def _hybrid_tensors(model):
    """(config, tensors on the host by name): values that bfloat16 holds."""
    g = _gen(23, len(model))
    if model == "vivezen":
        cfg = synth.hybrid_config(*HYBRIDS[model])
        names = {n: a.shape for n, a in _once("vivezen names", lambda: synth.hybrid_weights(cfg)).items()}
    else:
        cfg = synth.zufilorn_config(**ZUFILORN)
        names = {n: a.shape for n, a in _once("zufilorn names", lambda: synth.zufilorn_weights(cfg, ZUFILORN_RANK)).items()}
    plain = _kept[model + " names"]
    out = {}
    for n, s in names.items():
        leaf = n.rsplit(".", 1)[-1]
        if n == "embed":
            half = _normal(g, (s[0] + 1) // 2, s[1])
            sign = torch.where(torch.rand(s[1], generator=g, device="cuda") < 0.5, -1.0, 1.0)
            a = torch.stack([half, half * sign], 1).reshape(-1, s[1])[:s[0]]
        elif n == "final.norm":  # the picks' partners: by signs where the output is tied, by the head's order where it is not
            a = sign if model == "vivezen" else torch.zeros(s, device="cuda")
        elif n == "head":
            a = out["embed"].to("cuda").roll(7, 0) * s[1] ** -0.5
        elif len(s) == 2 and leaf not in ("conv", "mix"):
            a = _normal(g, *s, std=s[1] ** -0.5)
        elif leaf == "conv":
            a = _normal(g, *s, std=s[1] ** -0.5)
        elif leaf in ("lq1", "lk1", "lq2", "lk2"):
            a = _normal(g, *s, std=0.5 * s[0] ** -0.25)
        else:
            a = torch.from_numpy(np.ascontiguousarray(plain[n])).cuda()  # norms, decays, gates' biases, streams
        out[n] = a.bfloat16().float().cpu()
    return cfg, {n: a.numpy() for n, a in out.items()}


def _hybrid_model(model):
    return _once(model, lambda: b200nn.LanguageModel.from_weights(*_hybrid_tensors(model), _registry()))


# ---- a linear's weights: int4 in the layout the package takes ---------------------------------------
def _linear_numbers(shapes):
    """[(nibbles -8..7 [K, N], scales [groups, N], bias [N])] on the GPU, the same for every seed."""
    out = []
    for K, N in SHAPES[shapes]:
        g = _gen(31, K, N)
        q = torch.randint(-8, 8, (K, N), generator=g, device="cuda")
        s = (torch.rand((K + GROUP - 1) // GROUP, N, generator=g, device="cuda") * 0.015 + 0.005).half().float()
        out.append((q, s, _normal(g, N)))
    return out


def _linear_layers(shapes):
    def make():
        layers = []
        for (K, N), (q, s, b) in zip(SHAPES[shapes], _linear_numbers(shapes)):
            w = (q + 8).reshape(K // 8, 8, N) << (4 * torch.arange(8, device="cuda")).reshape(1, 8, 1)
            packed = w.sum(1).cpu().numpy().astype(np.uint32)
            layers.append(b200nn.Int4Linear(packed, s.cpu().numpy(), b.cpu().numpy(), K, N, GROUP, _registry()))
        return layers
    return _once("linear " + shapes, make)


def _linear_inputs(case, seed):
    return [_normal(_gen(seed, K, N), case["rows"], K) for K, N in SHAPES[case["shapes"]]]


# ---- attention's inputs ------------------------------------------------------------------------------
def _attention_inputs(case, seed):
    B, H = case["batch"], case["heads"]
    S, n = (1, case["ctx"]) if case["kind"] == "step_attention" else (case["seq"], case["past"] + case["seq"])
    g = _gen(seed, 41)
    q = _normal(g, B * S, H * 64).half()
    k, v = (_normal(g, B, H, n, 64).half() for _ in range(2))
    return q, k, v


def _prompts(case, seed, vocab):
    return np.random.Generator(np.random.PCG64([seed, 5])).integers(0, vocab, (case["batch"], case["prompt"])).astype(np.uint32)


def _requests(case, seed, vocab):
    """Token ids of every request: its prompt, then the tokens that follow one by one.  The lengths belong to the case."""
    lens = np.random.Generator(np.random.PCG64([case["requests"], case["longest"]])).integers(1, case["longest"] + 1, case["requests"])
    lens[0] = case["longest"]
    g = np.random.Generator(np.random.PCG64([seed, 7]))
    return [g.integers(0, vocab, int(n) + case["new"]).astype(np.uint32) for n in lens]


# ---- prepare and run ---------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        layers = _linear_layers(case["shapes"])
        xs = _linear_inputs(case, seed)
        ys = [torch.zeros(case["rows"], N, device="cuda") for _, N in SHAPES[case["shapes"]]]
        return {"case": case, "layers": layers, "x": xs, "y": ys}
    if kind in ("prompt_attention", "step_attention"):
        q, k, v = _attention_inputs(case, seed)
        return {"case": case, "reg": _registry(), "q": q, "k": k, "v": v, "out": torch.zeros_like(q)}
    if kind == "serve":
        model = _hybrid_model(case["model"])
        ids = _requests(case, seed, model.vocab_size)
        return {"case": case, "batch": b200nn.RequestBatch(model, len(ids), case["longest"] + case["new"]), "ids": ids}
    model = _gpt2_model(case["model"]) if kind == "gpt2" else _hybrid_model(case["model"])
    session = b200nn.DecodeSession(model, case["batch"], case["prompt"] + case["new"])
    return {"case": case, "session": session, "prompts": _prompts(case, seed, model.vocab_size)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        for layer, x, y in zip(state["layers"], state["x"], state["y"]):
            layer.forward_dev(x.data_ptr(), case["rows"], y.data_ptr())
        return state["y"]
    if kind == "prompt_attention":
        ops.prefill_attention_f16(state["q"].data_ptr(), state["k"].data_ptr(), state["v"].data_ptr(), case["batch"], case["heads"],
                                  case["past"] + case["seq"], case["seq"], case["past"], state["out"].data_ptr(), state["reg"])
        return state["out"]
    if kind == "step_attention":
        ops.decode_attention_f16(state["q"].data_ptr(), state["k"].data_ptr(), state["v"].data_ptr(), case["batch"], case["heads"], case["ctx"],
                                 case["ctx"], state["out"].data_ptr(), state["reg"])
        return state["out"]
    if kind == "serve":
        batch, ids, new = state["batch"], state["ids"], case["new"]
        out = [batch.step([(i, t[: len(t) - new], [len(t) - new - 1]) for i, t in enumerate(ids)])]
        for j in range(new):
            out.append(batch.step([(i, t[len(t) - new + j: len(t) - new + j + 1], [0]) for i, t in enumerate(ids)]))
        for i in range(len(ids)):
            batch.end(i)
        return out
    session = state["session"]
    session.prefill(state["prompts"])
    session.step(case["new"] - 1)
    return {"tokens": session.tokens().astype(np.int64), "logits": session.logits()}


# ---- what a pass cannot do without -------------------------------------------------------------------
def _gpt2_work(case):
    size, int4 = MODELS[case["model"]]
    cfg = getattr(b200nn.Gpt2Config, size)()
    B, S, new, d, L, V = case["batch"], case["prompt"], case["new"], cfg.n_embd, cfg.n_layer, cfg.vocab_size
    weights = 12 * d * d * L
    per = 0.5 + 2.0 / GROUP if int4 else 4.0
    steps = range(S, S + new - 1)  # positions before each step's token
    kv = 2 * d * 2 * L  # bytes of a cached position
    nbytes = new * (weights + V * d) * per + B * kv * (S + sum(p + 2 for p in steps)) + B * V * 4
    flops = 2.0 * B * (weights * (S + len(steps)) + V * d * new) + 4.0 * B * d * L * (S * (S + 1) / 2 + sum(p + 1 for p in steps))
    return {"bytes": nbytes, "flops": flops}


def _hybrid_sizes(cfg, rank):
    """(parameters of the layers, [(sequence flops a token, state values, cache values a position) of each layer])."""
    d, n, per_layer = cfg["width"], 0, []
    for layer in cfg["layers"]:
        x, ff = layer["mixer"], layer["mlp"]["ff"]
        H, dim, vd = x["heads"], x["dim"], x["vdim"]
        n += 3 * d * ff + d * H * vd
        if layer["type"] == "latent_attention":
            rd, R, Q = x["rot_dim"], x["kv_rank"], x["q_rank"]
            n += d * (Q + R + rd + H) + Q * H * (dim + rd) + R * H * (dim + vd)
            per_layer.append((0, 0, R + rd, 2 * H * (dim + rd + vd), x["mask"]["size"]))
        elif layer["type"] == "attention":
            G = x["kv_heads"]
            n += d * (2 * H * dim + G * (2 * dim + vd) + H)
            per_layer.append((0, 0, G * (2 * dim + vd), 4 * H * (dim + vd), 1 << 30))
        elif layer["type"] == "mlstm":
            n += d * H * (2 * dim + 2 * vd + 2)
            per_layer.append((4 * H * dim * vd, H * dim * (vd + 1), 0, 0, 0))
        else:
            KH = x["kv_heads"]
            n += d * (2 * KH * dim + H * vd + H)
            n += rank * (2 * d + H * (dim + vd)) if layer["type"] == "channel_delta" else d * (H + H * vd)
            per_layer.append((6 * H * dim * vd, H * dim * vd, 0, 0, 0))
    return n, per_layer


def _hybrid_work(cfg, rank, lens, new, picks):
    """lens: prompt lengths; new: single tokens after them; picks: rows whose logits are wanted."""
    params, layers = _hybrid_sizes(cfg, rank)
    d, V = cfg["width"], cfg["vocab"]
    tokens = sum(lens) + new * len(lens)
    nbytes = (1 + new) * (params + V * d) * 2.0 + picks * V * 4.0
    flops = 2.0 * params * tokens + 2.0 * V * d * picks
    for scan, state, row, pair, window in layers:
        flops += scan * tokens
        nbytes += len(lens) * state * 4.0 * (1 + 2 * new)
        for n in lens:
            seen = [min(p + 1, window) for p in range(n + new)]
            flops += pair * sum(seen)
            nbytes += row * 2.0 * (n + sum(seen[n:]) + new)
    return {"bytes": nbytes, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "linear":
        M = case["rows"]
        return {"bytes": sum(K * N / 2 + (K + GROUP - 1) // GROUP * N * 2 + N * 4 + M * (K + N) * 4 for K, N in SHAPES[case["shapes"]]),
                "flops": sum(2.0 * M * K * N for K, N in SHAPES[case["shapes"]])}
    if kind == "prompt_attention":
        B, H, S, past = case["batch"], case["heads"], case["seq"], case["past"]
        return {"bytes": B * H * 64 * 2.0 * (2 * S + 2 * (past + S)), "flops": 4.0 * 64 * B * H * (S * past + S * (S + 1) / 2)}
    if kind == "step_attention":
        B, H, n = case["batch"], case["heads"], case["ctx"]
        return {"bytes": B * H * 64 * 2.0 * (2 + 2 * n), "flops": 4.0 * 64 * B * H * n}
    if kind == "gpt2":
        return _gpt2_work(case)
    if kind == "hybrid":
        return _hybrid_work(synth.hybrid_config(*HYBRIDS[case["model"]]), 0, [case["prompt"]] * case["batch"], case["new"] - 1, case["batch"] * case["new"])
    lens = [len(t) - case["new"] for t in _requests(case, 0, 32000)]
    return _hybrid_work(synth.zufilorn_config(**ZUFILORN), ZUFILORN_RANK, lens, case["new"], len(lens) * (1 + case["new"]))


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":  # up to two rows multiply in 32 bits; more round activations and weights to fp16
        return {"rel": 1e-5} if case["rows"] <= 2 else {"rel": 1.2e-3}
    if kind in ("prompt_attention", "step_attention"):  # fp16 in and out: 2.8e-4 seen
        return {"rel": 1e-3}
    if kind == "gpt2":  # activations between Linears and the cache are fp16: 4.5e-4 of the logits seen
        return {"rel": 2e-3, "differ": 0.002}
    return {"rel": 0.03, "max": 0.5, "differ": 0.002}  # bfloat16 activations and weights: 8e-3 seen


# ---- the same in 64 bits -------------------------------------------------------------------------------
def _f64(a):
    return (torch.from_numpy(a).cuda() if isinstance(a, np.ndarray) else a).double()


def _softmax_attention(q, k, v, past, scale=0.125):
    """q [..., S, n] at positions past.., k and v [..., past + S, n]."""
    s = q @ k.transpose(-1, -2) * scale
    S, T = s.shape[-2:]
    at = torch.arange(T, device="cuda")
    s = s.masked_fill(at[None, :] > past + torch.arange(S, device="cuda")[:, None], -math.inf)
    return torch.softmax(s, -1) @ v


def _layer_norm(x, g, b, eps):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], g, b, eps)


def _gpt2_exact(case, seed):
    def make():
        cfg, w = _gpt2_tensors(case["model"])
        return cfg, {n: _f64(a) for n, a in w.items()}
    cfg, w = _once("exact " + case["model"], make)
    prompts = torch.from_numpy(_prompts(case, seed, cfg.vocab_size).astype(np.int64)).cuda()
    H, d, eps, new = cfg.n_head, cfg.n_embd, cfg.layer_norm_epsilon, case["new"]
    tokens, logits = [], []
    for ids in prompts.split(max(1, min(64, 16384 // case["prompt"]))):
        B, cap = len(ids), case["prompt"] + new
        cache = [torch.zeros(2, B, H, cap, 64, dtype=torch.float64, device="cuda") for _ in range(cfg.n_layer)]
        past, got = 0, []
        for _ in range(new):
            S = ids.shape[1]
            x = w["wte"][ids] + w["wpe"][past:past + S]
            for i in range(cfg.n_layer):
                p = f"h.{i % DISTINCT_LAYERS}."
                lin = lambda t, n: t @ w[p + n + ".weight"] + w[p + n + ".bias"]  # noqa: E731
                h = lin(_layer_norm(x, w[p + "ln_1.weight"], w[p + "ln_1.bias"], eps), "attn.c_attn")
                q, k, v = h.reshape(B, S, 3, H, 64).permute(2, 0, 3, 1, 4)
                cache[i][0, :, :, past:past + S], cache[i][1, :, :, past:past + S] = k, v
                a = _softmax_attention(q, cache[i][0, :, :, :past + S], cache[i][1, :, :, :past + S], past)
                x = x + lin(a.transpose(1, 2).reshape(B, S, d), "attn.c_proj")
                h = lin(_layer_norm(x, w[p + "ln_2.weight"], w[p + "ln_2.bias"], eps), "mlp.c_fc")
                x = x + lin(torch.nn.functional.gelu(h, approximate="tanh"), "mlp.c_proj")
            last = _layer_norm(x[:, -1], w["ln_f.weight"], w["ln_f.bias"], eps) @ w["wte"].T
            past += S
            ids = last.argmax(-1, keepdim=True)
            got.append(ids)
        tokens.append(torch.cat(got, 1))
        logits.append(last)
    return {"tokens": torch.cat(tokens), "logits": torch.cat(logits)}


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _unit(x):
    return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)


_silu, _softplus = torch.nn.functional.silu, torch.nn.functional.softplus


class _HybridExact:
    """A hybrid decoder over segments of tokens [B, T]; what a layer keeps between segments is in self.kept."""

    def __init__(self, cfg, w):
        self.cfg, self.w, self.kept, self.past = cfg, w, {}, 0

    def conv(self, key, x, w):
        taps = w.shape[1]
        before = self.kept.get(key)
        before = x.new_zeros(x.shape[0], taps - 1, x.shape[2]) if before is None else before
        xx = torch.cat([before, x], 1)
        self.kept[key] = xx[:, -(taps - 1):]
        return sum(xx[:, j:j + x.shape[1]] * w[:, j] for j in range(taps))

    def delta(self, i, h, x, w, channel):
        B, T, _ = h.shape
        H, KH, dim, vd = x["heads"], x["kv_heads"], x["dim"], x["vdim"]
        q, k, v = (_silu(self.conv((i, n), h @ w(n).T, w(n + ".conv"))) for n in "qkv")
        q = (_unit(q.reshape(B, T, KH, dim)) * dim ** -0.5).repeat_interleave(H // KH, 2)
        k = _unit(k.reshape(B, T, KH, dim)).repeat_interleave(H // KH, 2)
        v, beta = v.reshape(B, T, H, vd), torch.sigmoid(h @ w("b").T)
        if channel:
            z = _softplus(h @ w("a1").T @ w("a2").T + w("dt_bias")).reshape(B, T, H, dim)
            decay = torch.exp(-torch.exp(w("A_log"))[:, None] * z)
            gate = torch.sigmoid(h @ w("g1").T @ w("g2").T)
        else:
            decay = torch.exp(-torch.exp(w("A_log")) * _softplus(h @ w("a").T + w("dt_bias")))[..., None]
            gate = _silu(h @ w("g").T)
        S = self.kept.get(i)
        S = h.new_zeros(B, H, dim, vd) if S is None else S
        o = torch.empty(B, T, H, vd, dtype=h.dtype, device=h.device)
        for t in range(T):
            S = S * decay[:, t, :, :, None]
            u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhd,bhdv->bhv", k[:, t], S))
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            o[:, t] = torch.einsum("bhd,bhdv->bhv", q[:, t], S)
        self.kept[i] = S
        return (_rms(o, w("norm"), self.cfg["norm"]["eps"]) * gate.reshape(B, T, H, vd)).reshape(B, T, -1) @ w("o").T

    def mlstm(self, i, h, x, w):
        B, T, _ = h.shape
        H, dim, vd, cap = x["heads"], x["dim"], x["vdim"], x["gate_cap"]
        q, k = (h @ w("q").T).reshape(B, T, H, dim) * dim ** -0.5, (h @ w("k").T).reshape(B, T, H, dim)
        v = (h @ w("v").T).reshape(B, T, H, vd)
        gi = cap * torch.tanh((h @ w("i").T + w("i.b")) / cap)
        gf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w("f").T + w("f.b")) / cap))
        S, n, m = self.kept.get(i) or (h.new_zeros(B, H, dim, vd), h.new_zeros(B, H, dim), h.new_zeros(B, H))
        o = torch.empty(B, T, H, vd, dtype=h.dtype, device=h.device)
        for t in range(T):
            top = torch.maximum(gf[:, t] + m, gi[:, t])
            keep, write = torch.exp(gf[:, t] + m - top)[..., None], torch.exp(gi[:, t] - top)[..., None]
            n = keep * n + write * k[:, t]
            S = keep[..., None] * S + (write * k[:, t])[..., None] * v[:, t, :, None, :]
            m = top
            below = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            o[:, t] = torch.einsum("bhd,bhdv->bhv", q[:, t], S) / below[..., None]
        self.kept[i] = (S, n, m)
        return (_rms(o, 1.0, self.cfg["norm"]["eps"]).reshape(B, T, -1) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T

    def cached(self, key, new):
        old = self.kept.get(key)
        self.kept[key] = new if old is None else torch.cat([old, new], 1)
        return self.kept[key]

    def seen(self, T, window):
        d = (self.past + torch.arange(T, device="cuda"))[:, None] - torch.arange(self.past + T, device="cuda")[None, :]
        return (d >= 0) & (d < window)

    def rotate(self, x, rot, at):
        """x [B, T, ..., dims]: entry i with entry i + dims / 2."""
        n = rot["dims"]
        f = float(rot["base"]) ** (-2.0 * torch.arange(n // 2, dtype=torch.float64, device="cuda") / n)
        a = at.double()[:, None] * f[None, :]
        c, s = torch.cos(a), torch.sin(a)
        if x.dim() == 4:
            c, s = c[:, None], s[:, None]
        u, v = x[..., :n // 2], x[..., n // 2:]
        return torch.cat([u * c - v * s, v * c + u * s], -1)

    def latent(self, i, h, x, w):
        B, T, _ = h.shape
        eps = self.cfg["norm"]["eps"]
        H, dim, rd, vd, R = x["heads"], x["dim"], x["rot_dim"], x["vdim"], x["kv_rank"]
        at = self.past + torch.arange(T, device="cuda")
        q = (_rms(h @ w("dq").T, w("dq.norm"), eps) @ w("uq").T).reshape(B, T, H, dim + rd)
        q = torch.cat([q[..., :dim], self.rotate(q[..., dim:], x["rot"], at)], -1)
        ckr = h @ w("dkv").T
        row = torch.cat([_rms(ckr[..., :R], w("dkv.norm"), eps), self.rotate(ckr[..., R:], x["rot"], at)], -1)
        rows, seen = self.cached(i, row), self.seen(T, x["mask"]["size"])
        gate, o = torch.sigmoid(h @ w("g").T), []
        for n in range(H):
            k = torch.cat([rows[..., :R] @ w("uk").reshape(H, dim, R)[n].T, rows[..., R:]], -1)
            s = (q[:, :, n] @ k.transpose(1, 2) * x["scale"]).masked_fill(~seen, -math.inf)
            o.append(torch.softmax(s, -1) @ (rows[..., :R] @ w("uv").reshape(H, vd, R)[n].T) * gate[..., n:n + 1])
        return torch.cat(o, -1) @ w("o").T

    def diff(self, i, h, x, w):
        B, T, _ = h.shape
        H, G, dim, vd, cap = x["heads"], x["kv_heads"], x["dim"], x["vdim"], x["softcap"]
        at = (self.past + torch.arange(T, device="cuda")).double()
        temp = 1.0 + x["q_temp"]["coef"] * torch.log(torch.floor((at + 1.0) / x["q_temp"]["every"]) + 1.0)
        q = (h @ w("q").T).reshape(B, T, H, 2, dim) * temp[:, None, None, None]
        k = self.cached((i, "k"), (h @ w("k").T).reshape(B, T, G, 2, dim))
        v = self.cached((i, "v"), (h @ w("v").T).reshape(B, T, G, vd))
        lam = torch.exp(w("lq1") @ w("lk1")) - torch.exp(w("lq2") @ w("lk2")) + x["diff"]
        gate, seen, o = torch.sigmoid(h @ w("g").T), self.seen(T, 1 << 30), []
        for n in range(H):
            maps = []
            for j in (0, 1):
                s = cap * torch.tanh(q[:, :, n, j] @ k[:, :, n * G // H, j].transpose(1, 2) * x["scale"] / cap)
                maps.append(torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, :, n * G // H])
            o.append(_rms(maps[0] - lam * maps[1], 1.0, self.cfg["norm"]["eps"]) * (1.0 - x["diff"]) * gate[..., n:n + 1])
        return torch.cat(o, -1) @ w("o").T

    def forward(self, ids):
        """The residual stream [B, T, width] of the tokens."""
        cfg, w, T = self.cfg, self.w, ids.shape[1]
        eps, zuf = cfg["norm"]["eps"], "streams" in cfg
        x = w["embed"][ids]
        if zuf:
            xs = (x + w["pos"][self.past:self.past + T])[None].repeat(cfg["streams"], 1, 1, 1)
        for i, layer in enumerate(cfg["layers"]):
            p = f"l{i}."
            mix = {"delta": lambda h, m, g: self.delta(i, h, m, g, False), "channel_delta": lambda h, m, g: self.delta(i, h, m, g, True),
                   "mlstm": lambda h, m, g: self.mlstm(i, h, m, g), "latent_attention": lambda h, m, g: self.latent(i, h, m, g),
                   "attention": lambda h, m, g: self.diff(i, h, m, g)}[layer["type"]]
            act = _silu if zuf else lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
            parts = (lambda h: mix(h, layer["mixer"], lambda n: w[p + "mix." + n]),
                     lambda h: (act(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T)
            for j, part in enumerate(parts, 1):
                norm = w[p + f"norm{j}"]
                if zuf:
                    c = {n: w[f"{p}hc{j}.{n}"] for n in ("in", "out", "mix")}
                    y = part(_rms(torch.einsum("s,sbtd->btd", c["in"], xs), 1.0 + norm, eps))
                    xs = torch.einsum("st,sbnd->tbnd", c["mix"], xs) + c["out"][:, None, None, None] * y
                else:
                    x = x + part(_rms(x, norm, eps))
        self.past += T
        return xs.sum(0) if zuf else x

    def logits(self, x):
        zuf = "head" in self.w
        return _rms(x, self.w["final.norm"] + (1.0 if zuf else 0.0), self.cfg["norm"]["eps"]) @ self.w["head" if zuf else "embed"].T


def _hybrid_exact(case, seed):
    def make():
        cfg, w = _hybrid_tensors(case["model"])
        return cfg, {n: _f64(a) for n, a in w.items()}
    cfg, w = _once("exact " + case["model"], make)
    if case["kind"] == "serve":  # one batch of the longest length: what follows a request's end does not reach back
        ids = _requests(case, seed, cfg["vocab"])
        rows = np.zeros((len(ids), max(len(t) for t in ids)), dtype=np.int64)
        for r, t in zip(rows, ids):
            r[: len(t)] = t
        x = _HybridExact(cfg, w).forward(torch.from_numpy(rows).cuda())
        m = _HybridExact(cfg, w)
        first = torch.tensor([len(t) - case["new"] - 1 for t in ids], device="cuda")
        return [m.logits(x[torch.arange(len(ids), device="cuda"), first + j]) for j in range(case["new"] + 1)]
    ids = torch.from_numpy(_prompts(case, seed, cfg["vocab"]).astype(np.int64)).cuda()
    m, got = _HybridExact(cfg, w), []
    for _ in range(case["new"]):
        last = m.logits(m.forward(ids)[:, -1])
        ids = last.argmax(-1, keepdim=True)
        got.append(ids)
    return {"tokens": torch.cat(got, 1), "logits": last}


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        out = []
        for x, (q, s, b) in zip(_linear_inputs(case, seed), _linear_numbers(case["shapes"])):
            w = q.double() * s.double().repeat_interleave(GROUP, 0)[: len(q)]
            out.append(x.double() @ w + b.double())
        return out
    if kind in ("prompt_attention", "step_attention"):
        q, k, v = _attention_inputs(case, seed)
        B, H, n = k.shape[:3]
        S = q.shape[0] // B
        o = _softmax_attention(q.double().reshape(B, S, H, 64).transpose(1, 2), k.double(), v.double(), n - S)
        return o.transpose(1, 2).reshape(q.shape)
    if kind == "gpt2":
        return _gpt2_exact(case, seed)
    return _hybrid_exact(case, seed)
