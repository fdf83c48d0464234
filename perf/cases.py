"""The work whose speed this repository is measured by, through its public entry points: training steps of
the preset decoders (engine.TrainEngine), and serving (prompt passes, greedy generation, single chosen tokens)
of the presets and of the layer-list designs (engine.Decoder, engine.HybridDecoder).

A case is a dict of plain values:
  what    "train"     one optimizer step on rows x seq positions
          "generate"  prompt pass, then `new` greedy tokens
          "steps"     prompt pass, then `new` chosen tokens one by one, logits after each (a sampling client)
          "prefill"   prompt pass with the logits of eight rows
  model   a preset's name, or zutalix-SIZE / detatar-SIZE of serve_bench

Inputs are synthetic (uniform token ids, spans of supervised positions, random weights), all made from the
seed. Serving weights are drawn so that the next token is decided by a clear margin, as a trained model
decides it: embeddings about as strong as what the layers add, the untied head equal to the embedding.

`exact` restates the models in plain torch in 64 bits.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from emberlm_b200 import engine as E
from emberlm_b200 import lib
from emberlm_b200 import serve_bench as SB

HP = dict(lr=1e-4, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.01, clip=1.0)
MICRO = 4          # rows of a micro-batch where the rows divide by it
WANT = 8           # rows whose logits a prompt pass returns
F64 = torch.float64


# ---- cases --------------------------------------------------------------------------------------
def _train(model, rows, seq, precision="tf32", ckpt=False, **k):
    return {"what": "train", "model": model, "rows": rows, "seq": seq, "precision": precision, "checkpointing": ckpt, **k}


def _serve(what, model, prompt, new, **k):
    return {"what": what, "model": model, "prompt": prompt, "new": new, **k}


def listed():
    return [
        # one short conversation a step: every kernel is small, launches and dependences decide
        _train("smollm2_135m", 1, 127, name="train_135m_1x127"),
        # SmolLM2-135M on 4 x 512: the smallest of the benchmark's training workloads
        _train("smollm2_135m", 4, 511, name="train_135m_4x511"),
        # the same model where near-fp32 products are asked for, on ragged rows
        _train("smollm2_135m", 3, 301, "3xtf32", name="train_135m_3x301_3xtf32"),
        # two ranks' share of the benchmark's default workload (32 x 1024)
        _train("smollm2_360m", 16, 1023, name="train_360m_16x1023"),
        # one micro-batch of the QK-Norm, head size 128 model
        _train("qwen3_0_6b", 2, 2047, name="train_qwen3_0_6b_2x2047"),
        # one micro-batch with recomputation and llama3 rotary scaling
        _train("llama3_2_1b", 4, 2047, ckpt=True, name="train_llama3_1b_4x2047_ckpt"),
        # the benchmark's generation request, a quarter of its new tokens
        _serve("generate", "qwen3_0_6b", 256, 128, name="generate_qwen3_0_6b_256_128"),
        # a short chat turn of the smallest model
        _serve("generate", "smollm2_135m", 37, 48, name="generate_135m_37_48"),
        # a client that samples: logits come back after every token
        _serve("steps", "smollm2_360m", 700, 16, name="steps_360m_700_16"),
        # layer lists: a long prompt, and generation behind a short one, of either design
        _serve("prefill", "zutalix-0.6b", 4096, 0, name="prefill_zutalix_0_6b_4096"),
        _serve("generate", "zutalix-0.6b", 300, 64, name="generate_zutalix_0_6b_300_64"),
        _serve("generate", "detatar-0.6b", 1000, 64, name="generate_detatar_0_6b_1000_64"),
    ]


def draw(rng: random.Random):
    def logu(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    presets = ("smollm2_135m", "smollm2_360m", "qwen3_0_6b", "llama3_2_1b", "qwen3_1_7b")
    lists = ("zutalix-0.6b", "detatar-0.6b", "zutalix-1.7b", "detatar-1.7b")
    most = work(listed()[5])["flops"]
    what = rng.choice(("train", "train", "train", "generate", "generate", "steps", "prefill"))
    if what == "train":
        while True:
            model = rng.choice(presets)
            big = model in ("llama3_2_1b", "qwen3_1_7b")
            precision = "3xtf32" if not big and rng.random() < 0.15 else "tf32"
            c = _train(model, rng.randint(1, 16), logu(100, 2047), precision, big or rng.random() < 0.2)
            limit = 0.05 if precision == "3xtf32" else 1.0
            if c["rows"] * c["seq"] <= (8192 if model not in presets[:2] else 16384) and work(c)["flops"] <= limit * most:
                return c
    while True:
        model = rng.choice(presets + lists)
        prompt = logu(64, 4096) if what == "prefill" else logu(8, 2048)
        c = _serve(what, model, prompt, {"prefill": 0, "generate": logu(8, 128), "steps": logu(4, 24)}[what])
        if work(c)["bytes"] <= work(listed()[6])["bytes"]:
            return c


# ---- models -------------------------------------------------------------------------------------
def _is_preset(case):
    return case["model"] in E.PRESETS


def _preset_tensors(cfg):
    """(name, shape) of a preset's parameters in arena order."""
    hid, I, D = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    H, Hk = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    out = [("model.embed_tokens.weight", (cfg["vocab_size"], hid))]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        out += [(p + "input_layernorm.weight", (hid,)), (p + "self_attn.q_proj.weight", (H * D, hid)),
                (p + "self_attn.k_proj.weight", (Hk * D, hid)), (p + "self_attn.v_proj.weight", (Hk * D, hid)),
                (p + "self_attn.o_proj.weight", (hid, H * D))]
        if cfg.get("qk_norm"):
            out += [(p + "self_attn.q_norm.weight", (D,)), (p + "self_attn.k_norm.weight", (D,))]
        out += [(p + "post_attention_layernorm.weight", (hid,)), (p + "mlp.gate_proj.weight", (I, hid)),
                (p + "mlp.up_proj.weight", (I, hid)), (p + "mlp.down_proj.weight", (hid, I))]
    return out + [("model.norm.weight", (hid,))]


def _layer_list(model):
    """(config, {name: shape}) of a layer-list model."""
    family, size = model.split("-")
    preset = E.PRESETS[SB.SIZES[size][0]]
    if family == "zutalix":
        cfg = SB.zutalix_config(preset, SB.SIZES[size][1], preset["num_hidden_layers"])
        return cfg, SB.zutalix_shapes(cfg, SB.SIZES[size][1][5])
    cfg = SB.detatar_config(preset, size, preset["num_hidden_layers"])
    cfg["embedding"]["scale"] = float(cfg["width"]) ** 0.5
    return cfg, SB.detatar_shapes(cfg, SB.DETATAR_SIZES[size][1][2])


def _generator(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 16 + k)


def _preset_weights(case, seed):
    """Training: N(0, 0.02), as the benchmark starts from. Serving: stronger embeddings, and the matrices that
    write to the residual stream scaled down by the root of their number."""
    cfg, gen, out = E.PRESETS[case["model"]], _generator(seed), {}
    serve = case["what"] != "train"
    small = 0.02 / math.sqrt(2 * cfg["num_hidden_layers"])
    for name, shape in _preset_tensors(cfg):
        t = torch.empty(shape, device="cuda")
        if len(shape) == 1:
            t.normal_(1.0, 0.1, generator=gen)
        elif serve and name.startswith("model.embed"):
            t.normal_(0.0, 0.1, generator=gen)
        elif serve and name.endswith(("o_proj.weight", "down_proj.weight")):
            t.normal_(0.0, small, generator=gen)
        else:
            t.normal_(0.0, 0.02, generator=gen)
        out[name] = t
    return out


def _list_weights(model, seed):
    """bfloat16, as the weight files hold them."""
    cfg, shapes = _layer_list(model)
    gen, out = _generator(seed), {}
    post = (2 * len(cfg["layers"])) ** -0.5
    for name, shape in shapes.items():
        if name == "head":
            out[name] = out["embed"]
            continue
        t = torch.empty(shape, device="cuda", dtype=torch.bfloat16)
        last = name.rsplit(".", 1)[-1]
        if last in ("norm1b", "norm2b"):
            t.normal_(post, 0.1 * post, generator=gen)
        elif "norm" in last or last == "out":
            t.normal_(1.0, 0.1, generator=gen)
        elif last == "conv":
            t.normal_(0.0, 0.3, generator=gen)
        elif last == "shift" or ".mu." in name:
            t.uniform_(0.0, 1.0, generator=gen)
        elif last == "correction":
            t.normal_(0.0, 0.02, generator=gen)
        elif last in ("A_log", "dt_bias", "w0"):
            t.normal_(-1.0, 0.5, generator=gen)
        elif last in ("b", "u") and len(shape) == 1 or last == "u":
            t.normal_(0.0, 0.5, generator=gen)
        else:
            t.normal_(0.0, 0.02, generator=gen)
        out[name] = t
    return out


def _vocab(case):
    return E.PRESETS[case["model"]]["vocab_size"] if _is_preset(case) else _layer_list(case["model"])[0]["vocab"]


def _batch(case, seed):
    """ids, targets, mask [rows, seq]: uniform tokens, alternating spans of 16 to 128 supervised positions."""
    rows, seq = case["rows"], case["seq"]
    tok = torch.randint(0, _vocab(case), (rows, seq + 1), generator=_generator(seed, 1), device="cuda")
    rng, mask = random.Random(seed), np.zeros((rows, seq), np.float32)
    for r in range(rows):
        at, on = rng.randint(4, 32), True
        while at < seq:
            n = rng.randint(16, 128)
            if on:
                mask[r, at:at + n] = 1.0
            at, on = at + n, not on
    return tok[:, :-1].contiguous(), tok[:, 1:].contiguous(), torch.from_numpy(mask).cuda()


def _micro(case):
    return MICRO if case["rows"] % MICRO == 0 else case["rows"]


def _row_weights(case, mask):
    """mask / (sum of its micro-batch's mask x micro-batches)."""
    n = case["rows"] // _micro(case)
    m = mask.reshape(n, -1)
    return (m / (m.sum(1, keepdim=True) * n)).reshape(mask.shape).contiguous()


def _prompt(case, seed):
    return torch.randint(0, _vocab(case), (case["prompt"],), generator=_generator(seed, 1), device="cuda")


def _chosen(case, seed):
    rng = random.Random(seed)
    return [rng.randrange(_vocab(case)) for _ in range(case["new"])]


def _wanted(case):
    n = case["prompt"]
    return [n - 1 - (i * n) // WANT for i in reversed(range(WANT))]


# ---- the measured calls -------------------------------------------------------------------------
def prepare(case, seed):
    if case["what"] == "train":
        cfg = E.make_config(**E.PRESETS[case["model"]], gradient_checkpointing=case["checkpointing"],
                            precision=lib.GEMM_3XTF32 if case["precision"] == "3xtf32" else lib.GEMM_TF32)
        eng = E.TrainEngine(cfg, case["rows"], case["seq"], **HP)
        eng.load_parameters(_preset_weights(case, seed))
        ids, targets, mask = _batch(case, seed)
        active = mask.reshape(-1).nonzero().reshape(-1).to(torch.int32)
        return {"case": case, "engine": eng, "batch": (ids, targets, mask, _row_weights(case, mask)), "active": active}
    context = (case["prompt"] + case["new"] + 1 + 127) // 128 * 128
    if _is_preset(case):
        dec = E.Decoder(E.make_config(**E.PRESETS[case["model"]]), context)
        dec.load_parameters(_preset_weights(case, seed))
    else:
        cfg, shapes = _layer_list(case["model"])
        dec = E.HybridDecoder(E.HybridModel(cfg, shapes), context)
        dec.load_parameters(_list_weights(case["model"], seed))
    return {"case": case, "decoder": dec, "prompt": _prompt(case, seed), "chosen": _chosen(case, seed)}


def run(state):
    case = state["case"]
    if case["what"] == "train":
        eng = state["engine"]
        eng.train_step(*state["batch"], active_rows=state["active"])
        # the loss is the engine's own memory, which ends with it: a logging client keeps a copy
        return {"loss_sums": eng.loss_sums.clone(), "params": eng.params, "grads": eng.grads, "m": eng.m, "v": eng.v}
    dec = state["decoder"]
    if case["what"] == "generate":
        return {"tokens": dec.generate(state["prompt"], case["new"]), "logits": dec.last_logits()}
    dec.reset()
    if case["what"] == "prefill":
        return {"logits": dec.extend(state["prompt"], _wanted(case))}
    logits = [dec.extend(state["prompt"], [case["prompt"] - 1])[0]]
    return {"logits": logits + [dec.step(t) for t in state["chosen"]]}


# ---- what a pass cannot do without ----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sizes(model):
    """(parameters a token multiplies with, of these in the head, bytes of one of them, attention width:
    sum over layers of score and value widths of all heads, cache bytes a position)"""
    if model in E.PRESETS:
        c = E.PRESETS[model]
        n = sum(math.prod(s) for _, s in _preset_tensors(c))
        L, D = c["num_hidden_layers"], c["head_dim"]
        return n, c["vocab_size"] * c["hidden_size"], 4, 2 * L * c["num_attention_heads"] * D, 8 * L * c["num_key_value_heads"] * D
    cfg, shapes = _layer_list(model)
    share = SB.TOP / (SB.EXPERTS + SB.IDENTITY)
    n = sum(math.prod(s) * (share if ".mlp.e" in k else 1.0) for k, s in shapes.items() if k != "embed")
    width = cache = 0
    for lay in cfg["layers"]:
        m = lay["mixer"]
        if lay["type"] == "parallel":
            a = m["left"]
            width += 2 * a["heads"] * a["dim"]
            cache += 4 * a["kv_heads"] * a["dim"]
        elif lay["type"] == "latent_attention":
            width += m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            cache += 2 * (m["kv_rank"] + m["rot_dim"])
    return n, cfg["vocab"] * cfg["width"], 2, width, cache


def _visible(case, T):
    """Sum over T positions of the keys each one sees."""
    size = 1024 if case["model"].startswith("zutalix") else T
    full, rest = divmod(T, size)
    return full * size * (size + 1) // 2 + rest * (rest + 1) // 2


def work(case):
    n, head, size, width, cache = _sizes(case["model"])
    if case["what"] == "train":
        tokens = case["rows"] * case["seq"]
        flops = 3 * (2.0 * tokens * (n - head / 2) + case["rows"] * width * _visible(case, case["seq"]) * 2.0)
        return {"bytes": 28.0 * n, "flops": flops}
    T, new = case["prompt"], case["new"]
    passes = 1 + max(0, new - (case["what"] == "generate"))
    flops = 2.0 * (n - head) * T + 2.0 * width * _visible(case, T) + 2.0 * (passes - 1) * (n + width * T)
    rows = WANT if case["what"] == "prefill" else passes
    return {"bytes": passes * (n * size + cache * T) + 4.0 * rows * _vocab(case), "flops": flops + 2.0 * head * rows}


def tolerance(case):
    if case["what"] == "train":
        # measured against `exact`: 2.7e-5 and 2.4e-3 (second moments have the largest error); single values
        # of a tensor scatter far more than the whole (measured between two runs: 4e-5 and 5e-2)
        return {"rel": 1.2e-4, "max": 1e-2} if case["precision"] == "3xtf32" else {"rel": 1e-2, "max": 0.3}
    # TF32 prompts of the presets: 9e-4; bfloat16 layer lists: 2.7e-3
    return {"rel": 4e-3, "differ": 0.0} if _is_preset(case) else {"rel": 1.2e-2, "differ": 0.0}


# ---- the same in 64 bits --------------------------------------------------------------------------
def _norm(x, w, eps, groups=1):
    parts = x.reshape(*x.shape[:-1], groups, -1)
    y = (parts * torch.rsqrt(parts.square().mean(-1, keepdim=True) + eps)).reshape(x.shape)
    return y if w is None else y * w


def _frequencies(dims, base, scaling=None, by_wavelength=False):
    """Inverse frequencies with wavelength-dependent scaling; the middle band is blended linearly in the
    frequency, or (the presets) in the wavelength."""
    out = []
    for i in range(dims // 2):
        f = base ** (-2.0 * i / dims)
        if scaling:
            wave, (factor, low, high, original) = 2 * math.pi / f, scaling
            if wave > original / low:
                f = f / factor
            elif wave >= original / high:
                s = (original / wave - low) / (high - low)
                if by_wavelength:
                    s = 1 - (wave - original / high) / (original / low - original / high)
                f = (1 - s) * f / factor + s * f
        out.append(f)
    return torch.tensor(out, dtype=F64, device="cuda")


def _turn(u, v, freqs):
    """The pairs (u, v) [T, ..., pairs] turned by position x frequency."""
    a = torch.arange(u.shape[0], dtype=F64, device="cuda")[:, None] * freqs
    a = a.reshape(u.shape[0], *([1] * (u.dim() - 2)), -1)
    return u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()


def _rotate_half(x, freqs):
    n = x.shape[-1] // 2
    return torch.cat(_turn(x[..., :n], x[..., n:], freqs), -1)


def _attend(q, k, v, scale):
    """Causal softmax attention of q [T, H, d] over k [T, G, d], v [T, G, dv]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    hidden = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
    out = []
    for g in range(G):
        s = torch.einsum("ihd,jd->hij", q[:, g * H // G:(g + 1) * H // G], k[:, g]) * scale
        out.append(torch.einsum("hij,jd->ihd", s.masked_fill(hidden, -math.inf).softmax(-1), v[:, g]))
    return torch.cat(out, 1)


def _preset_layer(x, w, cfg, freqs):
    """w: the layer's tensors in arena order."""
    D, H, Hk, eps, T = cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"], x.shape[0]
    w = iter(w)
    h = _norm(x, next(w), eps)
    q, k, v = (h @ next(w).T for _ in range(3))
    o = next(w)
    q, k, v = q.reshape(T, H, D), k.reshape(T, Hk, D), v.reshape(T, Hk, D)
    if cfg.get("qk_norm"):
        q, k = _norm(q, next(w), eps), _norm(k, next(w), eps)
    y = _attend(_rotate_half(q, freqs), _rotate_half(k, freqs), v, D ** -0.5)
    x = x + y.reshape(T, H * D) @ o.T
    h = _norm(x, next(w), eps)
    gate, up, down = next(w), next(w), next(w)
    return x + (torch.nn.functional.silu(h @ gate.T) * (h @ up.T)) @ down.T


def _preset_hidden(w, cfg, ids, keep):
    """Rows before the head. keep: whether a backward pass follows (layers are then recomputed in it)."""
    scaling = None
    if cfg.get("rope_scaling_factor"):
        scaling = tuple(cfg["rope_scaling_" + k] for k in ("factor", "low_freq_factor", "high_freq_factor", "original_max_pos"))
    freqs = _frequencies(cfg["head_dim"], cfg["rope_theta"], scaling, by_wavelength=True)
    per = (len(w) - 2) // cfg["num_hidden_layers"]
    x = w[0][ids].double()
    for i in range(cfg["num_hidden_layers"]):
        layer = [t.double() for t in w[1 + i * per:1 + (i + 1) * per]]
        x = checkpoint(_preset_layer, x, layer, cfg, freqs, use_reentrant=False) if keep else _preset_layer(x, layer, cfg, freqs)
    return _norm(x, w[-1].double(), cfg["rms_norm_eps"])


def _exact_step(case, seed):
    cfg = E.PRESETS[case["model"]]
    w = {k: t.double().requires_grad_() for k, t in _preset_weights(case, seed).items()}
    ids, targets, mask = _batch(case, seed)
    weight = _row_weights(case, mask.double())
    total = 0.0
    for r in range(case["rows"]):
        at = mask[r].nonzero().reshape(-1)
        if not len(at):
            continue
        logits = _preset_hidden(list(w.values()), cfg, ids[r], True)[at] @ w["model.embed_tokens.weight"].T
        loss = torch.nn.functional.cross_entropy(logits, targets[r, at], reduction="none")
        (loss * weight[r, at]).sum().backward()
        total += float(loss.detach().sum())
        del logits, loss
    grads = {k: t.grad for k, t in w.items()}
    norm = math.sqrt(sum(float(g.square().sum()) for g in grads.values()))
    scale = HP["clip"] / (norm + 1e-6) if norm > HP["clip"] else 1.0
    size = sum((t.numel() + 63) // 64 * 64 for t in w.values())
    out = {k: torch.zeros(size, dtype=F64, device="cuda") for k in ("params", "grads", "m", "v")}
    # the hyper-parameters are 32-bit numbers
    lr, b1, b2, eps, wd = (float(np.float32(HP[k])) for k in ("lr", "beta1", "beta2", "eps", "weight_decay"))
    at = 0
    for k, t in w.items():
        g, p = grads[k].reshape(-1), t.detach().reshape(-1)
        m, v = (1 - b1) * (g * scale), (1 - b2) * (g * scale).square()
        decay = wd if t.dim() == 2 else 0.0
        new = p - lr * ((m / (1 - b1)) / ((v / (1 - b2)).sqrt() + eps) + decay * p)
        for name, x in (("params", new), ("grads", g), ("m", m), ("v", v)):
            out[name][at:at + g.numel()] = x
        at += (g.numel() + 63) // 64 * 64
    return {"loss_sums": torch.tensor([total, float(mask.double().sum())], dtype=F64), **out}


def _previous(h):
    return torch.cat([torch.zeros_like(h[:1]), h[:-1]])


def _lightning(q, k, v, decay):
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device="cuda")
    decay, out = torch.tensor(decay, dtype=F64, device="cuda")[:, None, None], []
    for t in range(q.shape[0]):
        S = torch.baddbmm(decay * S, k[t, :, :, None], v[t, :, None, :])
        out.append(q[t, :, None, :] @ S)
    return torch.stack(out).squeeze(2)


def _delta_rule(q, k, v, g, beta):
    S, out = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device="cuda"), []
    for t in range(q.shape[0]):
        S = g[t, :, :, None] * S
        u = beta[t, :, None, None] * (v[t, :, None, :] - k[t, :, None, :] @ S)
        S = torch.baddbmm(S, k[t, :, :, None], u)
        out.append(q[t, :, None, :] @ S)
    return torch.stack(out).squeeze(2)


def _wkv_rule(r, k, v, decay, u):
    S, out = torch.zeros(r.shape[1], r.shape[2], v.shape[2], dtype=F64, device="cuda"), []
    for t in range(r.shape[0]):
        kv = k[t, :, :, None] * v[t, :, None, :]
        out.append(r[t, :, None, :] @ (S + u[:, :, None] * kv))
        S = decay[t, :, :, None] * S + kv
    return torch.stack(out).squeeze(2)


def _conv(x, taps):
    n, y = taps.shape[1], 0
    for j in range(n):
        back = n - 1 - j
        y = y + taps[:, j] * torch.cat([torch.zeros_like(x[:back]), x[:x.shape[0] - back]])
    return y


def _mix_parallel(h, w, p, m, eps):
    T, a, r, L, R = h.shape[0], m["left"], m["right"], p + "left.", p + "right."
    silu = torch.nn.functional.silu
    H, G, d = a["heads"], a["kv_heads"], a["dim"]
    q = (h @ w(L + "q").T + w(L + "q.b")).reshape(T, H, d)
    v = (h @ w(L + "k").T + w(L + "k.b")).reshape(T, G, d)
    s = a["rot"].get("scaling")
    freqs = _frequencies(a["rot"]["dims"], a["rot"]["base"], s and tuple(s[k] for k in ("factor", "low", "high", "original")))

    def rot(x):
        n = 2 * len(freqs)
        return torch.cat([torch.stack(_turn(x[..., 0:n:2], x[..., 1:n:2], freqs), -1).flatten(-2), x[..., n:]], -1)

    qr, kr, size = rot(q), rot(v), a["mask"]["size"]
    o = torch.cat([_attend(qr[i:i + size], kr[i:i + size], v[i:i + size], a["scale"]) for i in range(0, T, size)])
    left = (o * torch.sigmoid(h @ w(L + "g").T)[:, :, None]).reshape(T, H * d) @ w(L + "o").T
    H, d, dv = r["heads"], r["dim"], r["vdim"]
    q, k, v = (silu(h @ w(R + x).T).reshape(T, H, -1) for x in "qkv")
    o = _norm(_lightning(q, k, v, r["decay"]).reshape(T, H * dv), w(R + "norm"), eps) * torch.sigmoid(h @ w(R + "g").T)
    return 0.5 * (_norm(left, w(p + "left.out"), eps) + _norm(o @ w(R + "o").T, w(p + "right.out"), eps))


def _mix_delta(h, w, p, m, eps):
    T, H, G, d, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (torch.nn.functional.silu(_conv(h @ w(p + x).T, w(p + x + ".conv"))) for x in "qkv")
    q, k = (x.reshape(T, G, d) * torch.rsqrt(x.reshape(T, G, d).square().sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = (x.repeat_interleave(H // G, 1) for x in (q * d ** -0.5, k))
    z = (h @ w(p + "a1").T) @ w(p + "a2").T + w(p + "dt_bias")
    g = torch.exp(-torch.exp(w(p + "A_log"))[:, None] * torch.nn.functional.softplus(z, threshold=100).reshape(T, H, d))
    o = _norm(_delta_rule(q, k, v.reshape(T, H, dv), g, torch.sigmoid(h @ w(p + "b").T)), w(p + "norm"), eps)
    o = o * torch.sigmoid((h @ w(p + "g1").T) @ w(p + "g2").T).reshape(T, H, dv)
    return o.reshape(T, H * dv) @ w(p + "o").T


def _mix_latent(h, w, p, m, eps):
    T, H, d, dv, R = h.shape[0], m["heads"], m["dim"], m["vdim"], m["kv_rank"]
    freqs = _frequencies(m["rot_dim"], m["rot"]["base"])
    q = (_norm(h @ w(p + "dq").T, w(p + "dq.norm"), eps) @ w(p + "uq").T).reshape(T, H, -1)
    q = torch.cat([q[..., :d], _rotate_half(q[..., d:], freqs)], -1)
    down = h @ w(p + "dkv").T
    c, kr = _norm(down[:, :R], w(p + "dkv.norm"), eps), _rotate_half(down[:, R:], freqs)
    k = torch.cat([(c @ w(p + "uk").T).reshape(T, H, d), kr[:, None].expand(T, H, -1)], -1)
    o = _attend(q, k, (c @ w(p + "uv").T).reshape(T, H, dv), m["scale"]) * torch.sigmoid(h @ w(p + "g").T)[:, :, None]
    return o.reshape(T, H * dv) @ w(p + "o").T


def _mix_wkv(h, w, p, m, eps):
    T, H, d = h.shape[0], m["heads"], m["dim"]
    mixed = {s: h + (_previous(h) - h) * w(p + "mu." + s) for s in "rkvgw"}
    r, k, v = ((mixed[s] @ w(p + s).T).reshape(T, H, d) for s in "rkv")
    z = torch.tanh(mixed["w"] @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0")
    o = _norm(_wkv_rule(r, k, v, torch.exp(-torch.exp(z)).reshape(T, H, d), w(p + "u").reshape(H, d)), None, eps)
    return (o.reshape(T, H * d) * w(p + "norm") * torch.nn.functional.silu(mixed["g"] @ w(p + "g").T)) @ w(p + "o").T


def _glu(h, w, p, act):
    return (act(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T


def _experts(h, w, p, f):
    r, silu = f["router"], torch.nn.functional.silu
    s = (h @ w(p + "router").T).softmax(-1)
    choice = s + w(p + "correction")
    per = choice.shape[1] // r["groups"]["count"]
    best = choice.reshape(len(h), -1, per).amax(-1)
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(r["groups"]["keep"], 1).indices, True)
    chosen = choice.masked_fill(~kept.repeat_interleave(per, 1), -math.inf).topk(r["top"], 1).indices
    a = torch.zeros_like(s).scatter_(1, chosen, s.gather(1, chosen))
    a = a / (a.sum(1, keepdim=True) + 1e-20)
    out = h * a[:, r["experts"]:].sum(1, keepdim=True)
    for e in range(r["experts"]):
        rows = a[:, e].nonzero().reshape(-1)
        if len(rows):
            out[rows] += a[rows, e, None] * _glu(h[rows], w, f"{p}e{e}.", silu)
    return out + _glu(h, w, p + "shared.", silu) * torch.sigmoid(h @ w(p + "shared.sg").T)


def _list_hidden(cfg, weights, ids):
    def w(name):
        return weights[name].double()

    eps = cfg["norm"]["eps"]
    if cfg["architecture"] == "Zutalix":
        x = _norm(weights["embed"][ids].double(), w("embed.norm"), eps)
        for i, lay in enumerate(cfg["layers"]):
            p, mix = f"l{i}.", _mix_parallel if lay["type"] == "parallel" else _mix_delta
            x = x + _norm(mix(_norm(x, w(p + "norm1"), eps), w, p + "mix.", lay["mixer"], eps), w(p + "norm1b"), eps)
            h, limit = _norm(x, w(p + "norm2"), eps), lay["mlp"]["limit"]
            g, u = (h @ w(p + "mlp.gate").T).clamp(max=limit), (h @ w(p + "mlp.up").T).clamp(-limit, limit)
            x = x + _norm((g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(p + "mlp.down").T, w(p + "norm2b"), eps)
        return _norm(x, w("final.norm"), eps)
    groups = cfg["norm"]["groups"]
    x = weights["embed"][ids].double() * cfg["embedding"]["scale"]
    for i, lay in enumerate(cfg["layers"]):
        p, mix, f = f"l{i}.", _mix_latent if lay["type"] == "latent_attention" else _mix_wkv, lay["mlp"]
        h = _norm(x, w(p + "norm1"), eps, groups)
        y = mix(h + (_previous(h) - h) * w(p + "shift"), w, p + "mix.", lay["mixer"], eps)
        gelu = functools.partial(torch.nn.functional.gelu, approximate="tanh")
        ff = _glu(h, w, p + "mlp.", gelu) if f["kind"] == "dense" else _experts(h, w, p + "mlp.", f)
        x = x + y * torch.sigmoid(h @ w(p + "rg1").T + w(p + "rg1.b")) + ff * torch.sigmoid(h @ w(p + "rg2").T + w(p + "rg2.b"))
    return _norm(x, w("final.norm"), eps, groups)


def exact(case, seed):
    if case["what"] == "train":
        return _exact_step(case, seed)
    with torch.no_grad():
        if _is_preset(case):
            weights, cfg = _preset_weights(case, seed), E.PRESETS[case["model"]]
            head = weights["model.embed_tokens.weight"]

            def hidden(ids):
                return _preset_hidden(list(weights.values()), cfg, ids, False)
        else:
            weights, (cfg, _) = _list_weights(case["model"], seed), _layer_list(case["model"])
            head = weights["head"]

            def hidden(ids):
                return _list_hidden(cfg, weights, ids)

        head, prompt, n = head.double(), _prompt(case, seed), case["prompt"]
        if case["what"] == "prefill":
            return {"logits": hidden(prompt)[_wanted(case)] @ head.T}
        if case["what"] == "steps":
            ids = torch.cat([prompt, torch.tensor(_chosen(case, seed), device="cuda")])
            return {"logits": list(hidden(ids)[n - 1:] @ head.T)}
        # greedy tokens by guessing all of them and correcting the guess until it stands
        tokens = prompt[-1:].expand(case["new"])
        for _ in range(4):
            logits = hidden(torch.cat([prompt, tokens[:-1]]))[n - 1:] @ head.T
            if torch.equal(logits.argmax(-1), tokens):
                return {"tokens": None, "logits": logits[-1]}
            tokens = logits.argmax(-1)
        return None
