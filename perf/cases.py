"""
Performance cases: what a user has this framework do, through its public entry points, from the smallest call to the
largest. A case is a dict of plain values; `prepare` makes what a program holds before the call, `run` is one pass.

  kind "prompt"   a prompt through `Engine.open_sequence(...).extend(...)`: the last position's logits and what the cache holds
  kind "decode"   rows of one prompt continued token by token with the model's captured step (`runtime`), tokens given:
                  every step's logits and the cache
  kind "train"    `TrainStep.step`: forward, backward and the MuonAdamW update on `accum` micro-batches: loss, weights, momenta

GPT cases are named by depth as the training script derives them (width 64 x depth rounded up to whole heads of 128, vocabulary
32768, sequence length 2048); Lupodra and Safepel by width and layers with the layers of `scripts/serve_bench.py`.
"""

import math

import torch
import torch.nn.functional as F

VOCAB, SEQ, HEAD = 32768, 2048, 128
PAGE = 64                              # tokens of a cache page
EPS = 2.0 ** -23                       # RMS norm of GPT
BF16 = torch.bfloat16
LR_SCALE = 0.02                        # where the learning-rate schedule stands


def listed():
    return [
        # the smallest model answering one user: every launch of the step counts
        dict(name="decode_d4_1row", kind="decode", model="GPT", depth=4, rows=1, prompt=19, steps=32, pattern="SSSL"),
        # chat with the speedrun model: one row, a prompt of ordinary length behind it
        dict(name="decode_d26_1row", kind="decode", model="GPT", depth=26, rows=1, prompt=512, steps=16, pattern="SSSL"),
        # several samples of one prompt (evaluation by sampling, RL rollouts)
        dict(name="decode_d26_8rows", kind="decode", model="GPT", depth=26, rows=8, prompt=512, steps=16, pattern="SSSL"),
        # the widest step the captured path takes
        dict(name="decode_d26_64rows", kind="decode", model="GPT", depth=26, rows=64, prompt=512, steps=16, pattern="SSSL"),
        # the served families, as their benchmark runs them
        dict(name="decode_lupodra_8rows", kind="decode", model="Lupodra", width=1664, layers=26, rows=8, prompt=512, steps=16),
        dict(name="decode_safepel_3rows", kind="decode", model="Safepel", width=1664, layers=26, rows=3, prompt=300, steps=16),
        # a short question to a small model: bound by launches; a long document to the speedrun model: bound by arithmetic
        dict(name="prompt_d12_45", kind="prompt", model="GPT", depth=12, tokens=45, pattern="SSSL"),
        dict(name="prompt_d26_2000", kind="prompt", model="GPT", depth=26, tokens=2000, pattern="SSSL"),
        dict(name="prompt_safepel_1111", kind="prompt", model="Safepel", width=768, layers=12, tokens=1111),
        # the toy run of the quick start, pretraining at the reference depth, and the speedrun recipe's device batch
        dict(name="train_d4", kind="train", depth=4, batch=8, length=512, accum=1, fp8=False, pattern="SSSL"),
        dict(name="train_d12_bf16", kind="train", depth=12, batch=32, length=2048, accum=1, fp8=False, pattern="SSSL"),
        dict(name="train_d26_fp8", kind="train", depth=26, batch=16, length=2048, accum=1, fp8=True, pattern="SSSL"),
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "train"])
    pattern = rng.choice(["SSSL", "SSSL", "SSSL", "L"])
    if kind == "train":
        most = _train_tokens_cost(dict(depth=26, batch=16, length=2048, accum=1))
        while True:
            case = dict(kind="train", depth=rng.randrange(4, 27, 2), batch=_log_uniform(rng, 1, 32), length=_log_uniform(rng, 100, 2048),
                        accum=rng.choice([1, 1, 2]), fp8=rng.random() < 0.4, pattern=pattern)
            if _train_tokens_cost(case) <= most:
                return case
    model = rng.choice(["GPT", "GPT", "GPT", "Safepel", "Lupodra"])
    if model == "GPT":
        case = dict(kind=kind, model=model, depth=rng.randrange(4, 27, 2), pattern=pattern)
    else:
        case = dict(kind=kind, model=model, width=128 * rng.randrange(2, 14), layers=rng.randrange(2, 27, 2))
    if kind == "decode":
        return dict(case, rows=_log_uniform(rng, 1, 64), prompt=_log_uniform(rng, 2, 1900), steps=rng.randrange(8, 33))
    return dict(case, tokens=_log_uniform(rng, 2, 2040))


# ------------------------------------------------------------------------------------ sizes, work

def _width(depth):
    return -(-depth * 64 // HEAD) * HEAD


def _gpt_matmul_params(depth):
    C = _width(depth)
    return 12 * C * C * depth + VOCAB * C


def _train_tokens_cost(case):
    return case["batch"] * case["length"] * case["accum"] * _gpt_matmul_params(case["depth"])


def _has_ve(i, depth):
    return i % 2 == (depth - 1) % 2


def _windows(case):
    """Tokens a query of each layer looks back over (its own not counted); SEQ: all."""
    n, pattern = case["depth"], case["pattern"]
    short = -(-SEQ // 4 // 128) * 128
    sizes = [SEQ if pattern[i % len(pattern)] == "L" else short for i in range(n)]
    sizes[-1] = SEQ
    return sizes


def _pairs(n, window, start=0):
    """(query, key) pairs of queries start .. start + n - 1."""
    return sum(min(t, window) + 1 for t in range(start, start + n))


def _gpt_work(case, queries, start, rows):
    """FLOPs of the forward pass over `queries` positions of `rows` rows and the attention's share of keys and values."""
    C, depth = _width(case["depth"]), case["depth"]
    pairs = [_pairs(queries, w, start) for w in _windows(case)]
    return rows * (2 * _gpt_matmul_params(depth) * queries + 4 * C * sum(pairs)), rows * 4 * C * sum(pairs)


def _served_sizes(case):
    C, L = case["width"], case["layers"]
    if case["model"] == "Safepel":
        return 12 * C * C * L + VOCAB * C, 12 * C * C * L + VOCAB * C
    per_dense = 2 * C * C + 1.4 * C * C + 2 * C * C + 8 * C * C
    token, stored = per_dense + C * C * 4, per_dense + 48 * C * C - 8 * C * C
    return (per_dense + token) / 2 * L + VOCAB * C, (per_dense + stored) / 2 * L + VOCAB * C


def work(case):
    if case["kind"] == "train":
        tokens, P = case["batch"] * case["length"] * case["accum"], _gpt_matmul_params(case["depth"])
        C = _width(case["depth"])
        pairs = sum(_pairs(case["length"], w) for w in _windows(case)) * case["batch"] * case["accum"]
        tables = (1 + case["depth"] // 2) * VOCAB * C
        return {"bytes": 16.0 * P + 12.0 * tables + 16 * tokens, "flops": 6.0 * P * tokens + 12.0 * C * pairs}
    if case["model"] == "GPT":
        P = _gpt_matmul_params(case["depth"])
        C = _width(case["depth"])
        if case["kind"] == "prompt":
            flops, _ = _gpt_work(case, case["tokens"], 0, 1)
            return {"bytes": 2.0 * P + 4.0 * C * case["depth"] * case["tokens"], "flops": flops - 2.0 * VOCAB * C * (case["tokens"] - 1)}
        flops, kv = _gpt_work(case, case["steps"], case["prompt"], case["rows"])
        return {"bytes": 2.0 * P * case["steps"] + kv + 4.0 * VOCAB * case["rows"] * case["steps"], "flops": flops}
    token, stored = _served_sizes(case)
    if case["kind"] == "prompt":
        return {"bytes": 2.0 * stored, "flops": 2.0 * token * case["tokens"]}
    touched = min(stored, token + (stored - token) * min(1.0, case["rows"] / 4))
    return {"bytes": (2.0 * touched + 4.0 * VOCAB * case["rows"]) * case["steps"], "flops": 2.0 * token * case["rows"] * case["steps"]}


# ------------------------------------------------------------------------------------ weights

class _Values:
    """Random tensors in a fixed order from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, shape, std):
        return torch.randn(shape, generator=self.g, device="cuda").mul_(std)

    def uniform(self, shape, lo, hi):
        return torch.rand(shape, generator=self.g, device="cuda").mul_(hi - lo).add_(lo)

    def ids(self, shape):
        return torch.randint(0, VOCAB, shape, generator=self.g, device="cuda")


def _gpt_tensors(case, v):
    """A GPT some way into training: the scales of its initialisation, output projections and scalars that have moved off zero."""
    depth = case["depth"]
    C, H = _width(depth), _width(depth) // HEAD
    b = (3.0 / C) ** 0.5
    t = {"transformer.wte.weight": v.normal((VOCAB, C), 0.8).to(BF16), "lm_head.weight": v.normal((VOCAB, C), 0.05)}
    for i in range(depth):
        p = f"transformer.h.{i}."
        for n in ("c_q", "c_k", "c_v"):
            t[p + f"attn.{n}.weight"] = v.uniform((C, C), -b, b)
        t[p + "attn.c_proj.weight"] = v.uniform((C, C), -0.5 * b, 0.5 * b)
        t[p + "mlp.c_fc.weight"] = v.uniform((4 * C, C), -0.6 * b, 0.6 * b)
        t[p + "mlp.c_proj.weight"] = v.uniform((C, 4 * C), -0.5 * b, 0.5 * b)
        if _has_ve(i, depth):
            t[p + "attn.ve_gate.weight"] = v.uniform((H, 12), -0.3, 0.3)
            t[f"value_embeds.{i}.weight"] = v.uniform((VOCAB, C), -b, b).to(BF16)
    t["resid_lambdas"] = 1.0 + v.uniform((depth,), 0.0, 0.1)
    t["x0_lambdas"] = v.uniform((depth,), 0.05, 0.2)
    t["smear_gate.weight"] = v.uniform((1, 24), -0.1, 0.1)
    t["smear_lambda"] = v.uniform((1,), 0.2, 0.4)
    t["backout_lambda"] = v.uniform((1,), 0.15, 0.25)
    return t


def _lupodra_config(C, layers):
    mixer = {"heads": C // HEAD, "dim": HEAD, "rot_dim": 64, "vdim": HEAD, "kv_rank": 512, "q_rank": -(-C * 3 // 4 // 64) * 64,
             "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}, "mask": {"size": 512}}
    dense = {"kind": "dense", "ff": 4 * C}
    moe = {"kind": "moe", "expert": {"ff": C}, "router": {"experts": 16, "top": 4}}
    return {"architecture": "Lupodra", "vocab": VOCAB, "width": C, "norm": {"eps": 1e-6}, "residual_mult": 0.7, "loop": None,
            "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": moe if i % 2 else dense} for i in range(layers)]}


def _safepel_config(C, layers):
    heads = C // HEAD
    keys = max(k for k in range(1, heads // 2 + 1) if heads % k == 0)
    delta = {"heads": heads, "kv_heads": keys, "dim": HEAD, "vdim": HEAD, "conv": 4}
    a, b = heads - heads // 2, heads // 2
    left = {"heads": a, "kv_heads": 1, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "softcap": 20.0, "rot": {"base": 10000.0, "dims": HEAD},
            "mask": {"size": 512}}
    right = {"heads": b, "dim": HEAD, "vdim": HEAD, "decay": [1 - 2.0 ** -(2 + 6 * i / b) for i in range(b)]}
    mixers = [("delta", delta), ("parallel", {"left": left, "right": right, "left_scale": 0.7, "right_scale": 0.7})]
    return {"architecture": "Safepel", "vocab": VOCAB, "width": C, "norm": {"eps": 1e-6}, "logit_scale": 1.0,
            "layers": [{"type": mixers[i % 2][0], "mixer": mixers[i % 2][1], "mlp": {"kind": "dense", "ff": -(-C * 8 // 3 // 64) * 64}}
                       for i in range(layers)]}


def _served_config(case):
    return (_lupodra_config if case["model"] == "Lupodra" else _safepel_config)(case["width"], case["layers"])


def _served_shapes(model, cfg):
    C, out = cfg["width"], {"embed": (VOCAB, cfg["width"]), "final.norm": (cfg["width"],)}
    if model == "Safepel":
        out.update({"embed.norm": (C,), "head": (VOCAB, C)})
    for i, spec in enumerate(cfg["layers"]):
        m, f, l, x = spec["mixer"], spec["mlp"], f"l{i}.", f"l{i}.mix."
        out[l + "norm1"] = (C,)
        if model == "Lupodra":
            H = m["heads"]
            out.update({l + "rg1": (C, C), l + "rg1.b": (C,), l + "rg2": (C, C), l + "rg2.b": (C,), x + "dq": (m["q_rank"], C),
                        x + "dq.norm": (m["q_rank"],), x + "uq": (H * (m["dim"] + m["rot_dim"]), m["q_rank"]),
                        x + "dkv": (m["kv_rank"] + m["rot_dim"], C), x + "dkv.norm": (m["kv_rank"],), x + "uk": (H * m["dim"], m["kv_rank"]),
                        x + "uv": (H * m["vdim"], m["kv_rank"]), x + "o": (C, H * m["vdim"])})
            if f["kind"] == "dense":
                out.update({l + "mlp.up": (f["ff"], C), l + "mlp.down": (C, f["ff"]), l + "mlp.act": (4,)})
            else:
                out[l + "mlp.router"] = (f["router"]["experts"], C)
                for e in range(f["router"]["experts"]):
                    n = f["expert"]["ff"]
                    out.update({f"{l}mlp.e{e}.gate": (n, C), f"{l}mlp.e{e}.up": (n, C), f"{l}mlp.e{e}.down": (C, n)})
            continue
        out.update({l + "norm1b": (C,), l + "norm2": (C,), l + "norm2b": (C,), l + "mlp.gate": (f["ff"], C), l + "mlp.up": (f["ff"], C),
                    l + "mlp.down": (C, f["ff"])})
        if spec["type"] == "delta":
            H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for n, rows in (("q", G * d), ("k", G * d), ("v", H * e)):
                out.update({x + n: (rows, C), x + n + ".conv": (rows, m["conv"])})
            out.update({x + "b": (H, C), x + "a": (H, C), x + "A_log": (H,), x + "dt_bias": (H,), x + "norm": (e,), x + "g": (H * e, C),
                        x + "o": (C, H * e)})
        else:
            a, b = m["left"], m["right"]
            n = b["heads"] * HEAD
            out.update({x + "left.q": (a["heads"] * HEAD, C), x + "left.k": (HEAD, C), x + "left.o": (C, a["heads"] * HEAD), x + "right.q": (n, C),
                        x + "right.k": (n, C), x + "right.v": (n, C), x + "right.g": (n, C), x + "right.o": (C, n), x + "right.norm": (n,)})
    return out


def _served_tensors(case, v):
    """bf16 weights of a trained model's scales, norms near one."""
    out = {}
    for name, shape in _served_shapes(case["model"], _served_config(case)).items():
        if name.endswith("mlp.act"):
            w = 0.3 + v.normal(shape, 0.2)
        elif name.endswith("A_log"):
            w = -1.5 + v.normal(shape, 1.0)
        elif name.endswith("dt_bias"):
            w = -2.0 + v.normal(shape, 1.0)
        elif len(shape) == 1:                     # Lupodra stores the deviation from one, except inside its mixer
            near = 0.0 if case["model"] == "Lupodra" and not name.endswith(("dq.norm", "dkv.norm")) else 1.0
            w = near + v.normal(shape, 0.1)
        else:
            w = v.normal(shape, 1.0 if name == "embed" else shape[1] ** -0.5)
        out[name] = w.to(BF16)
    return out


# ------------------------------------------------------------------------------------ what a program holds

def _gpt(case, tensors):
    from nanochat_b200.models.gpt import GPT, GPTConfig
    C = _width(case["depth"])
    with torch.device("meta"):
        model = GPT(GPTConfig(sequence_len=SEQ, vocab_size=VOCAB, n_layer=case["depth"], n_head=C // HEAD, n_kv_head=C // HEAD, n_embd=C,
                              window_pattern=case["pattern"]))
    model.to_empty(device="cuda")
    model.init_weights()                          # the rotary tables; the weights come from `tensors`
    model.load_state_dict(tensors, strict=True)
    return model


def _served(case, tensors):
    from nanochat_b200.models import lupodra, safepel
    kind, config = {"Lupodra": (lupodra.Lupodra, lupodra.LupodraConfig), "Safepel": (safepel.Safepel, safepel.SafepelConfig)}[case["model"]]
    return kind(config.from_dict(_served_config(case), sequence_len=4096)).load_tensors(tensors, "cuda")


def _inference_model(case, v):
    if case["model"] == "GPT":
        return _gpt(case, _gpt_tensors(case, v)).eval()
    return _served(case, _served_tensors(case, v)).eval()


def prepare(case, seed):
    v = _Values(seed)
    return {"train": _prepare_train, "decode": _prepare_decode, "prompt": _prepare_prompt}[case["kind"]](case, v)


def _prepare_prompt(case, v):
    from nanochat_b200.engine import Engine
    tokens = v.ids((case["tokens"],)).tolist()
    state = dict(case=case, engine=Engine(_inference_model(case, v), None), tokens=tokens)
    run(state)                                    # a served model has answered before
    return state


def _prepare_decode(case, v):
    from nanochat_b200 import runtime
    from nanochat_b200.engine import PagedKVCache
    prompt, ids = v.ids((1, case["prompt"])), v.ids((case["rows"], case["steps"]))
    model = _inference_model(case, v)
    with torch.inference_mode():
        if case["model"] == "GPT":
            cfg = model.config
            cache = PagedKVCache(batch_size=case["rows"], num_heads=cfg.n_kv_head, seq_len=cfg.sequence_len, head_dim=HEAD,
                                 num_layers=cfg.n_layer, device=model.get_device(), dtype=BF16)
        else:
            cache = model.make_cache(case["rows"])
        cache.reserve(case["prompt"], case["steps"])
        view = cache.begin_prompt(case["prompt"])
        model.forward(prompt, kv_cache=view)
        graph = getattr(runtime, getattr(model, "step_graph", "DecodeGraph"))(model, cache)
    state = dict(case=case, cache=cache, view=view, graph=graph, ids=[ids[:, t:t + 1].contiguous() for t in range(case["steps"])])
    run(state)                                    # the step is captured by now
    return state


def _prepare_train(case, v):
    from nanochat_b200 import ops
    from nanochat_b200.fp8 import Float8LinearConfig, convert_to_float8_training, default_fp8_filter
    from nanochat_b200.train import TrainStep
    shape = (case["batch"], case["length"] + 1)
    tokens = [v.ids(shape) for _ in range(case["accum"])]
    model = _gpt(case, _gpt_tensors(case, v))
    if case["fp8"]:
        convert_to_float8_training(model, config=Float8LinearConfig.from_recipe_name("tensorwise"), module_filter_fn=default_fp8_filter)
    trainer = TrainStep(model, grad_accum=case["accum"], weight_decay=0.1)
    for g in trainer.optimizer.param_groups:      # the end of the schedule
        g["lr"] = LR_SCALE * g["initial_lr"]
    batches = [(t[:, :-1].contiguous(), t[:, 1:].contiguous()) for t in tokens]
    return dict(case=case, trainer=trainer, batches=batches, native=ops.native_module())


# ------------------------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    if case["kind"] == "train":
        state["native"].set_fp8(case["fp8"])
        trainer = state["trainer"]
        loss = trainer.step(lambda i: state["batches"][i])
        model, optimizer = trainer.model, trainer.optimizer
        groups = model._arena.muon_groups
        out = {"loss": loss, "matrices": [g["master"] for g in groups], "lm_head": model.lm_head.weight,
               "tables": [model.transformer.wte.weight] + [e.weight for e in model.value_embeds.values()],
               "scalars": [model.resid_lambdas, model.x0_lambdas, model.smear_lambda, model.backout_lambda]}
        if not case["fp8"]:                       # 8-bit gradients: two right implementations differ by a tenth
            out["momenta"] = [optimizer.state[g["params"][0]]["momentum_buffer"] for g in groups]
            out["lm_head_avg"] = optimizer.state[model.lm_head.weight]["exp_avg"]
            out["scalars"].append(model.smear_gate.weight)
        return out
    if case["kind"] == "prompt":
        seq = state["engine"].open_sequence(case["tokens"] + 1)
        logits = seq.extend(state["tokens"], want=[case["tokens"] - 1])
        seq.close()
        return {"logits": logits, **_held(case, seq.cache, -(-case["tokens"] // PAGE))}
    with torch.inference_mode():
        state["cache"].fork(state["view"])
        state["graph"].begin()
        logits = [state["graph"].step(ids).clone() for ids in state["ids"]]
        return {"logits": torch.stack(logits), **_held(case, state["cache"], None)}


def _held(case, cache, pages):
    """What the cache holds: the prompt's pages, or everything."""
    if case["model"] == "GPT":
        return {"keys": cache.k_pool[:, :pages], "values": cache.v_pool[:, :pages]}
    out = {"store": [p[:pages] for p in cache.pools if p.shape[2]]}
    if case["model"] == "Safepel":
        out["states"] = cache.memory
    return out


# ------------------------------------------------------------------------------------ tolerance

def tolerance(case):
    """bf16 activations through the whole model. Measured with another attention implementation, worst output: prompts 0.0096 (largest
    0.053), bf16 training 0.014 (momenta; largest 0.14), fp8 training 0.015 (tables, where Adam takes the sign of a small gradient;
    largest 0.11); against 64 bits: 0.007 to 0.02."""
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.03, "max": 0.2}


# ------------------------------------------------------------------------------------ 64 bits

def _norm64(x, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _half_turn64(x, c, s):
    a, b = x.chunk(2, -1)
    return torch.cat([a * c + b * s, b * c - a * s], -1)


def _gpt64(case, W, ids, keep=None):
    """Logits before the soft cap's loss, (R, T, V), for (R, T) ids; `keep` collects each layer's keys and values."""
    depth, C = case["depth"], _width(case["depth"])
    R, T = ids.shape
    H = C // HEAD
    angle = torch.arange(T, device="cuda").float()[:, None] * (1.0 / (100000 ** (torch.arange(0, HEAD, 2, device="cuda").float() / HEAD)))
    cos, sin = angle.cos().to(BF16).double()[:, None], angle.sin().to(BF16).double()[:, None]     # the model's tables are bf16
    gap = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    e = _norm64(F.embedding(ids, W["transformer.wte.weight"]))
    gate = W["smear_lambda"] * torch.sigmoid(e[:, 1:, :24] @ W["smear_gate.weight"].T)
    x = x0 = torch.cat([e[:, :1], e[:, 1:] + gate * e[:, :-1]], 1)
    back = None
    for i, window in enumerate(_windows(case)):
        p = f"transformer.h.{i}."
        x = W["resid_lambdas"][i] * x + W["x0_lambdas"][i] * x0
        h = _norm64(x)
        q, k, v = (F.linear(h, W[p + f"attn.{n}.weight"]).view(R, T, H, HEAD) for n in ("c_q", "c_k", "c_v"))
        if _has_ve(i, depth):
            g = 3 * torch.sigmoid(h[..., :12] @ W[p + "attn.ve_gate.weight"].T)
            v = v + g[..., None] * F.embedding(ids, W[f"value_embeds.{i}.weight"]).view(R, T, H, HEAD)
        q, k = (1.2 * _norm64(_half_turn64(t, cos, sin)) for t in (q, k))
        if keep is not None:
            keep.append((k, v))
        score = torch.einsum("rihd,rjhd->rhij", q, k) * HEAD ** -0.5
        score = score.masked_fill((gap < 0) | (gap > window), -math.inf)
        y = torch.einsum("rhij,rjhd->rihd", torch.softmax(score, -1), v).reshape(R, T, C)
        x = x + F.linear(y, W[p + "attn.c_proj.weight"])
        x = x + F.linear(F.relu(F.linear(_norm64(x), W[p + "mlp.c_fc.weight"])).square(), W[p + "mlp.c_proj.weight"])
        if i == depth // 2:
            back = x
    return _norm64(x - W["backout_lambda"] * back)


def _cap64(x, W):
    return 15.0 * torch.tanh(F.linear(x, W["lm_head.weight"]) / 15.0)


def _operands64(tensors):
    """Matrices as the products read them (bf16), in 64 bits; vectors and small gates as they are."""
    return {n: (t if n.endswith("lambdas") or "gate" in n or t.numel() < 64 else t.to(BF16)).double() for n, t in tensors.items()}


def _safepel64(cfg, P, ids):
    T, eps = ids.numel(), cfg["norm"]["eps"]

    def ln(x, w):
        d = x - x.mean(-1, keepdim=True)
        return d * torch.rsqrt(d.square().mean(-1, keepdim=True) + eps) * w

    def rms(x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w

    def scan(decay, k, v, q, beta=None):
        S, out = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=torch.float64, device="cuda"), torch.empty_like(v)
        for t in range(T):
            S = S * decay[t][:, None, None]
            u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None]
            out[t] = torch.einsum("hde,hd->he", S, q[t])
        return out

    def delta(h, p, m):
        H, G, d = m["heads"], m["kv_heads"], m["dim"]

        def conv(n):
            w = P[p + n + ".conv"].double()
            x = F.pad(h @ P[p + n].double().T, (0, 0, m["conv"] - 1, 0))
            return F.silu(sum(w[:, j] * x[j:j + T] for j in range(m["conv"])))

        unit = lambda x: x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)
        q, k = (unit(conv(n).view(T, G, d)).repeat_interleave(H // G, 1) for n in ("q", "k"))
        beta = torch.sigmoid(h @ P[p + "b"].double().T)
        z = h @ P[p + "a"].double().T + P[p + "dt_bias"].double()
        decay = torch.exp(-torch.exp(P[p + "A_log"].double()) * F.softplus(z, threshold=40.0))
        o = rms(scan(decay, k, conv("v").view(T, H, -1), q * d ** -0.5, beta), P[p + "norm"].double())
        return (o.reshape(T, -1) * F.silu(h @ P[p + "g"].double().T)) @ P[p + "o"].double().T

    def parallel(h, p, m):
        a, b = m["left"], m["right"]
        i = torch.arange(HEAD // 2, device="cuda").double()
        angle = torch.arange(T, device="cuda").double()[:, None] * a["rot"]["base"] ** (-2 * i / HEAD)
        c, s = angle.cos()[:, None], angle.sin()[:, None]

        def turn(x):
            u, v = x[..., 0::2], x[..., 1::2]
            return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

        q, k = ((h @ P[p + "left." + n].double().T).view(T, -1, HEAD) for n in ("q", "k"))
        score = torch.einsum("ihd,jd->hij", turn(q), turn(k)[:, 0]) * a["scale"]
        gap = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
        score = (a["softcap"] * torch.tanh(score / a["softcap"])).masked_fill((gap < 0) | (gap >= a["mask"]["size"]), -math.inf)
        left = torch.einsum("hij,jd->ihd", torch.softmax(score, -1), k[:, 0]).reshape(T, -1) @ P[p + "left.o"].double().T
        q, k, v = (F.silu(h @ P[p + "right." + n].double().T).view(T, b["heads"], HEAD) for n in ("q", "k", "v"))
        decay = torch.tensor(b["decay"], dtype=torch.float64, device="cuda").expand(T, -1)
        y = rms(scan(decay, k, v, q).reshape(T, -1), P[p + "right.norm"].double()) * torch.sigmoid(h @ P[p + "right.g"].double().T)
        return m["left_scale"] * left + m["right_scale"] * (y @ P[p + "right.o"].double().T)

    x = ln(P["embed"][ids].double(), P["embed.norm"].double())
    for i, spec in enumerate(cfg["layers"]):
        n = lambda name: P[f"l{i}.{name}"].double()
        x = x + ln((delta if spec["type"] == "delta" else parallel)(ln(x, n("norm1")), f"l{i}.mix.", spec["mixer"]), n("norm1b"))
        h = ln(x, n("norm2"))
        x = x + ln((F.relu(h @ n("mlp.gate").T) * (h @ n("mlp.up").T)) @ n("mlp.down").T, n("norm2b"))
    return ln(x, P["final.norm"].double())


def _lupodra64(cfg, P, ids):
    T, eps = ids.numel(), cfg["norm"]["eps"]
    D = lambda name: P[name].double()
    n = lambda x: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    gap = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    x = D("embed")[ids]
    for i, spec in enumerate(cfg["layers"]):
        l, m, f = f"l{i}.", spec["mixer"], spec["mlp"]
        p, H, half = l + "mix.", m["heads"], m["rot_dim"] // 2
        angle = torch.arange(T, device="cuda").double()[:, None] * m["rot"]["base"] ** (-torch.arange(half, device="cuda").double() / half)

        def turn(z):
            c, s = (t.view(T, *([1] * (z.dim() - 2)), half) for t in (angle.cos(), angle.sin()))
            u, v = z[..., :half], z[..., half:]
            return torch.cat([u * c - v * s, v * c + u * s], -1)

        h = n(x) * (1 + D(l + "norm1"))
        q = ((n(h @ D(p + "dq").T) * D(p + "dq.norm")) @ D(p + "uq").T).view(T, H, -1)
        down = h @ D(p + "dkv").T
        c = n(down[:, :m["kv_rank"]]) * D(p + "dkv.norm")
        k, v = (c @ D(p + "uk").T).view(T, H, -1), (c @ D(p + "uv").T).view(T, H, -1)
        score = torch.einsum("ihd,jhd->hij", q[..., :m["dim"]], k) + torch.einsum("ihd,jd->hij", turn(q[..., m["dim"]:]), turn(down[:, m["kv_rank"]:]))
        score = (score * m["scale"]).masked_fill((gap < 0) | (gap >= m["mask"]["size"]), -math.inf)
        y = torch.einsum("hij,jhd->ihd", torch.softmax(score, -1), v).reshape(T, -1) @ D(p + "o").T
        change = torch.sigmoid(h @ D(l + "rg1").T + D(l + "rg1.b")) * y
        if f["kind"] == "dense":
            z, (a, b, d, e) = h @ D(l + "mlp.up").T, D(l + "mlp.act").unbind()
            ff = (a * n(z) + b * n(z * z) + d * n(z * z * z) + e) @ D(l + "mlp.down").T
        else:
            best, who = torch.topk(h @ D(l + "mlp.router").T, f["router"]["top"], -1)
            share = torch.zeros(T, f["router"]["experts"], dtype=torch.float64, device="cuda").scatter(1, who, torch.softmax(best, -1))
            ff = 0
            for j in range(f["router"]["experts"]):
                r = f"{l}mlp.e{j}."
                ff = ff + share[:, j:j + 1] * ((F.silu(h @ D(r + "gate").T) * (h @ D(r + "up").T)) @ D(r + "down").T)
        x = x + cfg["residual_mult"] * (change + torch.sigmoid(h @ D(l + "rg2").T + D(l + "rg2.b")) * ff)
    return n(x) * (1 + D("final.norm"))


def _served64(case, v):
    """Last hidden rows (after the final norm) and the output matrix for each row of ids."""
    P, cfg = _served_tensors(case, v), _served_config(case)
    body = _safepel64 if case["model"] == "Safepel" else _lupodra64
    out = P["head" if case["model"] == "Safepel" else "embed"].double()
    return lambda ids: body(cfg, P, ids), out


def exact(case, seed):
    v = _Values(seed)
    with torch.no_grad():
        if case["kind"] == "train":
            return _exact_train(case, v)
        if case["kind"] == "prompt":
            ids = v.ids((case["tokens"],))
            if case["model"] != "GPT":
                body, out = _served64(case, v)
                return {"logits": body(ids)[-1:] @ out.T}
            W, keep = _operands64(_gpt_tensors(case, v)), []
            logits = _cap64(_gpt64(case, W, ids[None], keep)[0, -1:], W)
            paged = lambda t: F.pad(t[0], (0, 0, 0, 0, 0, -case["tokens"] % PAGE)).unflatten(0, (-1, PAGE))
            return {"logits": logits, "keys": torch.stack([paged(k) for k, _ in keep]), "values": torch.stack([paged(x) for _, x in keep])}
        prompt, ids = v.ids((1, case["prompt"])), v.ids((case["rows"], case["steps"]))
        if case["model"] == "GPT":
            W = _operands64(_gpt_tensors(case, v))
            body, head = lambda one: _cap64(_gpt64(case, W, one[None])[0, case["prompt"]:], W), None
        else:
            inner, out = _served64(case, v)
            body = lambda one: inner(one)[case["prompt"]:] @ out.T
            if case["model"] == "Safepel" and case["rows"] * (case["prompt"] + case["steps"]) * case["layers"] > 100_000:
                return None                       # token by token in 64 bits: minutes
        return {"logits": torch.stack([body(torch.cat([prompt[0], row])) for row in ids], 1)}


POLAR = ((8.156554524902461, -22.48329292557795, 15.878769915207462), (4.042929935166739, -2.808917465908714, 0.5000178451051316),
         (3.8916678022926607, -2.772484153217685, 0.5060648178503393), (3.285753657755655, -2.3681294933425376, 0.46449024233003106),
         (2.3465413258596377, -1.7097828382687081, 0.42323551169305323))


def _muon64(g, w, lr, wd, beta2=0.9, momentum=0.95):
    """First Muon step on one matrix: (new weights, momentum)."""
    r, c = g.shape
    m = (1 - momentum) * g
    X = (1 - momentum) * g + momentum * m
    X = X * (X.norm() / r ** 0.5) / X.norm(dim=1, keepdim=True).clamp_min(1e-6)
    X = X / (X.norm() * 1.01 + 1e-6)
    X = X.T if r > c else X
    for a, b, d in POLAR:
        A = X @ X.T
        X = a * X + (b * A + d * (A @ A)) @ X
    X = X.T if r > c else X
    X = X * (min(r, c) ** 0.5 / X.norm().clamp_min(1e-6))
    dim = 1 if r >= c else 0
    mean, n = X.square().mean(dim, keepdim=True), X.shape[dim]
    step = ((1 - beta2) * mean).clamp_min(1e-10).rsqrt()
    X = X * step * ((mean.sum() * n).sqrt() / (mean * n * step.square()).sum().sqrt().clamp_min(1e-10))
    lr = lr * max(1.0, r / c) ** 0.5
    return w - lr * X - lr * wd * w * (X * w >= 0), m


def _adam64(g, w, lr, wd):
    """First AdamW step: the bias-corrected moments are g and g^2."""
    return w * (1 - lr * wd) - lr * g / (g.abs() + 1e-10)


def _exact_train(case, v):
    C, depth = _width(case["depth"]), case["depth"]
    tokens = [v.ids((case["batch"], case["length"] + 1)) for _ in range(case["accum"])]
    if case["fp8"] or work(case)["flops"] > 8e13:
        return None                               # rounded to 8 bits on purpose; or minutes in 64 bits
    masters = _gpt_tensors(case, v)
    W = {n: t.requires_grad_() for n, t in _operands64(masters).items()}
    rows_at_once = max(1, int(4e9 / (8 * case["length"] * (case["length"] * (C // HEAD) * 4 + 40 * C) * depth)))
    for t in tokens:
        total = 0.0
        for part in t.split(rows_at_once):
            with torch.enable_grad():
                logits = _cap64(_gpt64(case, W, part[:, :-1]), W)
                loss = F.cross_entropy(logits.flatten(0, 1), part[:, 1:].flatten(), reduction="sum") / (case["batch"] * case["length"])
                (loss / case["accum"]).backward()
            total += loss.item()
            del logits, loss
    s = LR_SCALE * (C / 768) ** -0.5
    names = [n for i in range(depth) for n in [f"transformer.h.{i}.attn.{m}.weight" for m in ("c_q", "c_k", "c_v", "c_proj")]
             + ([f"transformer.h.{i}.attn.ve_gate.weight"] if _has_ve(i, depth) else [])
             + [f"transformer.h.{i}.mlp.{m}.weight" for m in ("c_fc", "c_proj")]]
    matrices, momenta = [], []
    for shape in sorted({masters[n].shape for n in names}):
        new = [_muon64(W[n].grad, masters[n].double(), 0.02 * LR_SCALE, 0.1) for n in names if masters[n].shape == shape]
        matrices.append(torch.stack([a for a, _ in new]))
        momenta.append(torch.stack([b for _, b in new]))
    adam = lambda n, lr, wd: _adam64(W[n].grad, masters[n].double(), lr, wd)
    tables = [adam("transformer.wte.weight", 0.2 * s, 0.001)]
    tables += [adam(f"value_embeds.{i}.weight", 0.1 * s, 0.01) for i in range(depth) if _has_ve(i, depth)]
    scalars = [adam("resid_lambdas", 0.005 * LR_SCALE, 0.05), adam("x0_lambdas", 0.5 * LR_SCALE, 0.0)]
    scalars += [adam(n, 0.2 * LR_SCALE, 0.0) for n in ("smear_lambda", "backout_lambda", "smear_gate.weight")]
    return {"loss": total, "matrices": matrices, "momenta": momenta, "lm_head": adam("lm_head.weight", 0.004 * s, 0.01),
            "lm_head_avg": 0.2 * W["lm_head.weight"].grad, "tables": tables, "scalars": scalars}
