"""Workloads that stand for what this framework is used for, with the exact results they are held against.

A case is a dict of plain values.  ``kind`` says what is called:

* ``decode``: one recurrent step of the Taylor linear attention, ``ops.linattn_decode`` (the decode microbenchmark).
* ``linattn`` / ``window``: ``ops.linattn_prefill`` / ``ops.swa_prefill`` over whole sequences (the prefill sweep).
* ``mixer``: the ``LinearAttention`` module on a prompt, with its projections (the single-mixer configuration, in float32).
* ``prompt``: a whole model reads a prompt through ``advance`` and leaves its logits and its states.
* ``step``: a whole model decodes one token per sequence; the step is captured in a CUDA graph once, as ``generate(cg=True)``
  does it, and a pass is one replay.

``stack`` names the model: the Based model at its two sizes and the Razesun and Vubenex stacks of the same size, with random
weights in bfloat16."""
import math

import torch

from based_b200 import ops
from based_b200.mixers import LinearAttention
from based_b200.model import BasedConfig
from based_b200.registry import build_model

KERNEL_SIZE = 3      # BaseConv
TAPS = 4             # the short convolutions of Razesun


# --------------------------------------------------------------------------- the cases

def listed():
    return [
        # the decode microbenchmark: 256 sequences, 16 heads, float32 states, bfloat16 inputs; bound by the states' traffic
        {"name": "decode 256x16", "kind": "decode", "B": 256, "H": 16, "dv": 64, "state": "float32"},
        # the middle of the prefill sweep, linear attention and sliding window
        {"name": "linattn 8x16x8192", "kind": "linattn", "B": 8, "H": 16, "L": 8192, "dv": 64, "dtype": "bfloat16"},
        {"name": "window 8x16x8192", "kind": "window", "B": 8, "H": 16, "L": 8192, "hd": 64, "window": 64, "dtype": "bfloat16"},
        # the single-mixer configuration, in float32 with its projections
        {"name": "mixer fp32 2x1024", "kind": "mixer", "B": 2, "L": 1024, "d": 1024, "H": 16, "dtype": "float32"},
        # a batch of prompts for the 360M model (the generation configuration), and one short prompt of odd length
        {"name": "based prompt 16x2048", "kind": "prompt", "stack": "based-360m", "B": 16, "L": 2048},
        {"name": "based prompt 1x999", "kind": "prompt", "stack": "based-360m", "B": 1, "L": 999},
        # decoding with the 360M model at the generation configuration's batch, and with the 1.4B model at one GPU's share
        {"name": "based step 16", "kind": "step", "stack": "based-360m", "B": 16, "pos": 2100},
        {"name": "based-1b step 8", "kind": "step", "stack": "based-1b", "B": 8, "pos": 4100},
        # the hybrid stack: two long prompts at once (few sequences, much of the machine idle in a recurrence), decoding a batch
        {"name": "razesun prompt 2x4096", "kind": "prompt", "stack": "razesun-360m", "B": 2, "L": 4096},
        {"name": "razesun step 16", "kind": "step", "stack": "razesun-360m", "B": 16, "pos": 2100},
        # the post-norm stack: one user's long prompt of odd length, and that user's decoding
        {"name": "vubenex prompt 1x6001", "kind": "prompt", "stack": "vubenex-360m", "B": 1, "L": 6001},
        {"name": "vubenex step 1", "kind": "step", "stack": "vubenex-360m", "B": 1, "pos": 6100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "linattn", "window", "mixer", "prompt", "prompt", "prompt", "step", "step", "step"])
    if kind == "decode":
        return {"kind": kind, "B": _log(rng, 1, 256), "H": rng.choice([8, 12, 16]), "dv": rng.choice([64, 112]),
                "state": rng.choice(["float32", "bfloat16"])}
    if kind in ("linattn", "window"):
        B, H = _log(rng, 1, 16), rng.choice([8, 12, 16])
        size = rng.choice([64, 64, 112])
        L = min(_log(rng, 100, 32768), 8 * 16 * 8192 * 64 // (B * H * size))
        c = {"kind": kind, "B": B, "H": H, "L": L, "dtype": "bfloat16"}
        return dict(c, dv=size) if kind == "linattn" else dict(c, hd=size, window=rng.choice([32, 64, 64, 128]))
    if kind == "mixer":
        return {"kind": kind, "B": rng.choice([1, 2, 4]), "L": _log(rng, 60, 2048), "d": rng.choice([512, 1024]), "H": rng.choice([8, 16]),
                "dtype": "float32"}
    if kind == "prompt":
        stack = rng.choice(["based-360m", "razesun-360m", "vubenex-360m"])
        B = _log(rng, 1, 16)
        return {"kind": kind, "stack": stack, "B": B, "L": min(_log(rng, 30, 8000 if stack == "based-360m" else 6000), 32768 // B // (1 if stack[0] == "b" else 2))}
    return {"kind": kind, "stack": rng.choice(["based-360m", "razesun-360m", "vubenex-360m"]), "B": _log(rng, 1, 32), "pos": _log(rng, 100, 6000)}


# --------------------------------------------------------------------------- models, weights, contexts

def _config(stack):
    """The config of a stack as a config file holds it.  Razesun and Vubenex have the Based model's width and depth: RG-LRU
    layers or constant-decay linear attention where that has BaseConv, gated delta (or constant decay again) where it has
    LinearAttention, latent (every second one reads the cache of the one before) or grouped attention where it has SlidingAttention."""
    name, size = stack.split("-")
    base = BasedConfig.based_360m() if size == "360m" else BasedConfig.based_1b()
    d, heads = base.n_embd, base.n_embd // 128
    if name == "based":
        c = {k: getattr(base, k) for k in ("n_embd", "n_layer", "n_head", "alt_mixer_layers", "alt_mixer_2_layers", "vocab_size")}
        return dict(c, architecture="Based")
    layers, own = [], None
    for i in range(base.n_layer):
        if name == "vubenex" and i in base.alt_mixer_2_layers:
            layer = {"type": "attention", "mixer": {"heads": heads, "kv_heads": max(heads // 4, 1), "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                                    "q_temp": {"coef": 0.1, "every": 1024}}}
        elif name == "vubenex":
            layer = {"type": "lightning", "mixer": {"heads": heads, "dim": 128, "vdim": 128,
                                                    "decay": [1 - 2.0 ** -(5 + 5 * h / heads) for h in range(heads)]}}
        elif i in base.alt_mixer_layers:
            layer = {"type": "delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": TAPS}}
        elif i in base.alt_mixer_2_layers:
            m = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 512, "kv_rank": 256, "scale": 192 ** -0.5,
                 "rot": {"base": 1e4, "dims": 64}}
            if own is None:
                own = i
            else:
                m["kv_from"], own = own, None
            layer = {"type": "latent_attention", "mixer": m}
        else:
            layer = {"type": "rglru", "mixer": {"width": d, "blocks": heads, "conv": TAPS}}
        layers.append(dict(layer, mlp={"kind": "dense", "ff": 2 * d}))
    c = {"vocab": base.padded_vocab_size, "width": d, "layers": layers, "norm": {"eps": 1e-6}}
    if name == "razesun":
        return dict(c, architecture="Razesun", residual_mult=0.5, logit_scale=1.0)
    return dict(c, architecture="Vubenex", embedding={"scale": d ** 0.5}, max_positions=8192, token_side={"dim": 64})


def _layers(cfg):
    """(type, sizes, width, MLP width) of every layer."""
    if cfg["architecture"] != "Based":
        return [(lay["type"], lay["mixer"], cfg["width"], lay["mlp"]["ff"]) for lay in cfg["layers"]]
    d, H = cfg["n_embd"], cfg["n_head"]
    kinds = {**{i: "linattn" for i in cfg["alt_mixer_layers"]}, **{i: "window" for i in cfg["alt_mixer_2_layers"]}}
    return [(kinds.get(i, "conv"), {"heads": H, "dim": d // H}, d, 2 * d) for i in range(cfg["n_layer"])]


def _vocab(cfg):
    return (cfg["vocab_size"] + 7) // 8 * 8 if cfg["architecture"] == "Based" else cfg["vocab"]


def _shapes(cfg):
    """name -> (shape, standard deviation, mean) of every tensor of a model, by the names ``load_tensors`` takes."""
    t, V = {}, _vocab(cfg)

    def put(name, *shape, std=None, mean=0.0):
        t[name] = (shape, shape[-1] ** -0.5 if std is None else std, mean)

    if cfg["architecture"] == "Based":
        W = cfg["n_embd"]
        put("transformer.embeddings.word_embeddings.weight", V, W, std=1.0)   # the initialisation of nn.Embedding
        put("transformer.ln_f.weight", W, std=0.1, mean=1.0)
        for i, (kind, m, _, ff) in enumerate(_layers(cfg)):
            p = f"transformer.layers.{i}."
            for n in ("norm1", "norm2"):
                put(p + n + ".weight", W, std=0.1, mean=1.0)
            if kind == "linattn":
                put(p + "mixer.proj_q.weight", 16 * m["heads"], W)
                put(p + "mixer.proj_k.weight", 16 * m["heads"], W)
                put(p + "mixer.proj_v.weight", W, W)
                put(p + "mixer.out_proj.weight", W, W)
            elif kind == "window":
                put(p + "mixer.Wqkv.weight", 3 * W, W)
                put(p + "mixer.out_proj.weight", W, W)
            else:
                put(p + "mixer.in_proj.weight", 4 * W, W)
                put(p + "mixer.in_proj.bias", 4 * W, std=0.1)
                put(p + "mixer.conv.conv.weight", 2 * W, 1, KERNEL_SIZE)
                put(p + "mixer.out_proj.weight", W, 2 * W)
                put(p + "mixer.out_proj.bias", W, std=0.1)
            put(p + "mlp.fc1.weight", 2 * ff, W)
            put(p + "mlp.fc2.weight", W, ff)
        return t
    W = cfg["width"]
    put("embed", V, W)
    put("final.norm", W, std=0.1, mean=1.0)
    if cfg["architecture"] == "Razesun":
        put("embed.norm", W, std=0.1, mean=1.0)
        put("head", V, W)
    else:
        put("pos", cfg["max_positions"], W, std=0.3)
        put("side.embed", V, len(cfg["layers"]) * cfg["token_side"]["dim"], std=1.0)
    for i, (kind, m, _, ff) in enumerate(_layers(cfg)):
        p = f"l{i}.mix."
        for n in ("norm1", "norm2"):
            put(f"l{i}.{n}", W, std=0.1, mean=1.0 if cfg["architecture"] == "Razesun" else 0.6)
        if kind == "delta":
            H, d, dv = m["heads"], m["dim"], m["vdim"]
            for n in "qkv":
                put(p + n, H * (dv if n == "v" else d), W)
                put(p + n + ".conv", H * (dv if n == "v" else d), TAPS, std=0.5, mean=0.3)
            put(p + "a", H, W)
            put(p + "b", H, W)
            put(p + "A_log", H, std=0.5)
            put(p + "dt_bias", H, std=0.5, mean=-4.0)
            put(p + "norm", dv, std=0.1, mean=1.0)
            put(p + "g", H * dv, W)
            put(p + "o", W, H * dv)
        elif kind == "rglru":
            R, nb = m["width"], m["blocks"]
            for x in "xy":
                put(p + x, R, W)
                put(p + x + ".b", R, std=0.1)
            put(p + "conv", R, TAPS)
            put(p + "conv.b", R, std=0.1)
            for x in ("ra", "ri"):
                put(p + x, nb, R // nb, R // nb)
                put(p + x + ".b", nb, R // nb, std=0.5)
            put(p + "lam", R, std=1.0, mean=-4.0)
            put(p + "o", W, R)
        elif kind == "latent_attention":
            H, d, rd, dv, qr, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["q_rank"], m["kv_rank"]
            put(p + "dq", qr, W)
            put(p + "dq.norm", qr, std=0.1, mean=1.0)
            put(p + "uq", H * (d + rd), qr)
            if m.get("kv_from") is None:
                put(p + "dkv", r + rd, W)
                put(p + "dkv.norm", r, std=0.1, mean=1.0)
            put(p + "uk", H * d, r)
            put(p + "uv", H * dv, r)
            put(p + "g", H, W)
            put(p + "o", W, H * dv)
        elif kind == "attention":
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            for n, rows in (("q", H * d), ("k", G * d), ("g", H * d)):
                put(p + n, rows, W)
            put(p + "o", W, H * d)
            put(p + "q.norm", d, std=0.2, mean=1.0)
            put(p + "k.norm", d, std=0.2, mean=1.0)
        else:
            H, d, dv = m["heads"], m["dim"], m["vdim"]
            for n, rows in (("q", H * d), ("k", H * d), ("v", H * dv), ("g", H * dv)):
                put(p + n, rows, W)
            put(p + "norm", H * dv, std=0.1, mean=1.0)
            put(p + "o", W, H * dv)
        put(f"l{i}.mlp.gate", ff, W)
        put(f"l{i}.mlp.up", ff, W)
        put(f"l{i}.mlp.down", W, ff)
        if cfg["architecture"] == "Vubenex":
            n = cfg["token_side"]["dim"]
            put(f"l{i}.side.gate", n, W)
            put(f"l{i}.side.proj", W, n)
            put(f"l{i}.side.norm", W, std=0.1, mean=0.4)
    return t


def _gen(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _weights(cfg, seed):
    g = _gen(seed)
    return {n: _randn(g, *shape).mul_(std).add_(mean) for n, (shape, std, mean) in _shapes(cfg).items()}


class _Tensors:
    """A dict of tensors with the interface of a weights file."""

    def __init__(self, t):
        self.t, self.used = t, set()

    def __contains__(self, name):
        return name in self.t

    def get(self, name, shape):
        x = self.t[name]
        if tuple(x.shape) != tuple(shape):
            raise ValueError(f"{name} is {tuple(x.shape)}, not {tuple(shape)}")
        self.used.add(name)
        return x

    def unused(self):
        return [n for n in self.t if n not in self.used]


def _taylor(x):
    x2 = (x.unsqueeze(-1) * x.unsqueeze(-2)).flatten(-2) / math.sqrt(2)
    return torch.cat([torch.ones_like(x[..., :1]), x / 2, x2 / 4], -1)


def _context(cfg, case, seed):
    """What a step finds: per layer the tensors that ``pos`` tokens left there, as plain tensors in the caches' layouts."""
    g, B, pos, out = _gen(seed + 7919), case["B"], case["pos"], []
    for kind, m, W, _ in _layers(cfg):
        if kind == "linattn":
            H, dv, n = m["heads"], m["dim"], 32
            phi = _taylor(_randn(g, B, H, n, 16, dtype=torch.float32))
            v = _randn(g, B, H, n, dv, dtype=torch.float32)
            s = pos / n
            out.append([(torch.einsum("bhnd,bhnf->bhdf", v, phi) * s ** 0.5).unsqueeze(2).bfloat16(), (phi.sum(2) * s)[:, :, None, None].bfloat16()])
        elif kind == "window":
            out.append([_randn(g, B, pos + 4, 2, m["heads"], m["dim"])])
        elif kind == "conv":
            out.append([_randn(g, B, 2 * W, KERNEL_SIZE)])
        elif kind == "delta":
            H, d, dv = m["heads"], m["dim"], m["vdim"]
            out.append([_randn(g, B, TAPS, 2 * H * d + H * dv), _randn(g, B, H, d, dv, dtype=torch.float32) * 0.3])
        elif kind == "rglru":
            out.append([_randn(g, B, TAPS, m["width"]), _randn(g, B, m["width"], dtype=torch.float32)])
        elif kind == "latent_attention":
            out.append([] if m.get("kv_from") is not None else [_randn(g, B, pos + 4, m["kv_rank"] + m["rot_dim"])])
        elif kind == "attention":
            G, d = m["kv_heads"], m["dim"]
            keys = _randn(g, B, pos + 4, G * d)
            keys[:, pos:] = 0
            factor = torch.zeros(B, G, (pos + 4 + 127) // 128 * 128, device="cuda")
            factor[..., :pos] = torch.rsqrt(keys[:, :pos].float().view(B, pos, G, d).square().mean(-1) + cfg["norm"]["eps"]).transpose(1, 2)
            out.append([keys, factor])
        else:
            out.append([_randn(g, B, m["heads"], m["dim"], m["vdim"], dtype=torch.float32) * 3])
    return out


def _states(ip, n_layers):
    """The per-layer state tensors of a state container, without the workspaces kept beside them."""
    out = []
    for i in range(n_layers):
        s = ip.key_value_memory_dict[i]
        if isinstance(s, dict):
            out.append([s[k] for k in ("ring", "state", "conv", "keys", "factor") if k in s])
        else:
            out.append(list(s) if isinstance(s, (tuple, list)) else [s])
    return out


def _tokens(cfg, case, seed):
    return torch.randint(0, _vocab(cfg), (case["B"], case.get("L", 1)), generator=_gen(seed + 104729), device="cuda")


# --------------------------------------------------------------------------- prepare, run

def _inputs(case, seed):
    g, k = _gen(seed), case["kind"]
    if k == "decode":
        B, H, dv, sd = case["B"], case["H"], case["dv"], getattr(torch, case["state"])
        return {"q": _randn(g, B, H, 16) / 4, "k": _randn(g, B, H, 16) / 4, "v": _randn(g, B, H, dv) / 4,
                "kv": (_randn(g, B, H, 1, dv, 273, dtype=torch.float32) * 0.02).to(sd), "ks": (_randn(g, B, H, 1, 1, 273, dtype=torch.float32) * 0.02).to(sd)}
    if k == "linattn":   # views into one packed projection, as the mixer makes them
        B, H, L, dv = case["B"], case["H"], case["L"], case["dv"]
        x = _randn(g, B, L, H * (32 + dv), dtype=getattr(torch, case["dtype"])) / 4
        q, kk, v = x.split([16 * H, 16 * H, dv * H], -1)
        return {"q": q.unflatten(-1, (H, 16)).transpose(1, 2), "k": kk.unflatten(-1, (H, 16)).transpose(1, 2), "v": v.unflatten(-1, (H, dv)).transpose(1, 2)}
    if k == "window":
        x = _randn(g, case["B"], case["L"], 3, case["H"], case["hd"], dtype=getattr(torch, case["dtype"]))
        return {"qkv": x}
    d, dt = case["d"], getattr(torch, case["dtype"])
    w = [_randn(g, n, d, dtype=dt) * d ** -0.5 for n in (16 * case["H"], 16 * case["H"], d, d)]
    return {"w": w, "x": _randn(g, case["B"], case["L"], d, dtype=dt)}


def prepare(case, seed):
    k = case["kind"]
    with torch.no_grad():
        if k in ("decode", "linattn", "window"):
            return dict(_inputs(case, seed), kind=k, window=case.get("window"))
        if k == "mixer":
            x = _inputs(case, seed)
            m = LinearAttention(case["d"], num_heads=case["H"], layer_idx=0, device="cuda", dtype=getattr(torch, case["dtype"])).eval()
            for lin, w in zip((m.proj_q, m.proj_k, m.proj_v, m.out_proj), x["w"]):
                lin.weight.copy_(w)
            from based_b200.generation import InferenceParams
            ip = InferenceParams(max_seqlen=case["L"], max_batch_size=case["B"])
            ip.key_value_memory_dict[0] = m.allocate_inference_cache(case["B"], case["L"], dtype=getattr(torch, case["dtype"]))
            return {"kind": k, "m": m, "ip": ip, "x": x["x"]}
        cfg = _config(case["stack"])
        model = build_model(cfg, device="cuda", dtype=torch.bfloat16).eval()
        model.load_tensors(_Tensors(_weights(cfg, seed)))
        tokens, B, n = _tokens(cfg, case, seed), case["B"], len(_layers(cfg))
        if k == "prompt":
            return {"kind": k, "model": model, "ip": model.new_inference_params(B, case["L"]), "tokens": tokens, "n": n}
        pos = case["pos"]
        ip = model.new_inference_params(B, pos + 4)
        ip.seqlen_offset = pos
        ip.lengths_per_sample.fill_(pos)
        context = _context(cfg, case, seed)

        def rewind():
            for own, given in zip(_states(ip, n), context):
                for t, s in zip(own, given):
                    t.copy_(s)

        def step():
            return model(tokens, inference_params=ip, num_last_tokens=1)

        rewind()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = step()
        rewind()
        # the model and the container stay alive with the graph that reads them
        return {"kind": k, "graph": graph, "model": model, "ip": ip, "tokens": tokens, "out": [logits, _states(ip, n)]}


@torch.inference_mode()
def run(state):
    k = state["kind"]
    if k == "decode":
        y = ops.linattn_decode(state["q"], state["k"], state["v"], state["kv"], state["ks"])
        return [y, state["kv"], state["ks"]]
    if k == "linattn":
        return list(ops.linattn_prefill(state["q"], state["k"], state["v"]))
    if k == "window":
        x = state["qkv"]
        return ops.swa_prefill(x[:, :, 0], x[:, :, 1], x[:, :, 2], state["window"])
    if k == "mixer":
        y = state["m"](state["x"], inference_params=state["ip"])
        return [y, *state["ip"].key_value_memory_dict[0]]
    if k == "prompt":
        ip = state["ip"]
        ip.reset(ip.max_seqlen, ip.max_batch_size)
        logits = state["model"].advance(state["tokens"], ip, num_last_tokens=1)
        return [logits, _states(ip, state["n"])]
    state["graph"].replay()
    return state["out"]


# --------------------------------------------------------------------------- work, tolerance

def work(case):
    """Bytes: inputs, weights and states that are read, and what is written, once each.  Operations: matrix products, attention
    and recurrences, two per multiply-add."""
    k, B = case["kind"], case["B"]
    if k == "decode":
        H, dv, s = case["H"], case["dv"], 4 if case["state"] == "float32" else 2
        return {"bytes": B * H * (2 * s * 273 * (dv + 1) + 2 * (32 + 2 * dv)), "flops": 4 * B * H * 273 * (dv + 1)}
    if k == "linattn":
        n, s = B * case["H"] * case["L"], 2 if case["dtype"] == "bfloat16" else 4
        return {"bytes": n * s * (32 + 2 * case["dv"]), "flops": 4 * n * 273 * (case["dv"] + 1)}
    if k == "window":
        n, s = B * case["H"] * case["L"], 2 if case["dtype"] == "bfloat16" else 4
        return {"bytes": n * s * 4 * case["hd"], "flops": 4 * n * (min(case["window"], case["L"]) + 1) * case["hd"]}
    if k == "mixer":
        n, d, H = B * case["L"], case["d"], case["H"]
        return {"bytes": 4 * (2 * n * d + 2 * d * d + 32 * H * d + B * H * 273 * (d // H + 1)),
                "flops": 2 * n * (2 * d * d + 32 * H * d) + 4 * n * H * 273 * (d // H + 1)}
    cfg = _config(case["stack"])
    shapes, tables = _shapes(cfg), {"pos", "side.embed"} | ({"embed"} if cfg["architecture"] == "Razesun" else set())
    head = {"Based": "transformer.embeddings.word_embeddings.weight", "Razesun": "head", "Vubenex": "embed"}[cfg["architecture"]]
    size = {n: math.prod(s) for n, (s, _, _) in shapes.items()}
    matrices = sum(v for n, v in size.items() if n not in tables and n != head and len(shapes[n][0]) > 1)
    L = case.get("L", 1)
    flops, state = 2.0 * matrices * B * L + 2.0 * size[head] * B, 0
    past = case.get("pos", 0)
    seen = L * past + L * (L + 1) / 2   # keys seen by all tokens of a sequence
    for kind, m, W, _ in _layers(cfg):
        if kind == "linattn":
            flops += 4 * B * L * m["heads"] * 273 * (m["dim"] + 1)
            state += B * m["heads"] * 273 * (m["dim"] + 1) * 2 * (2 if past else 1)
        elif kind == "window":
            flops += 4 * B * L * 65 * W
            state += B * W * 2 * 2 * (66 if past else L)
        elif kind == "conv":
            state += B * 2 * W * KERNEL_SIZE * 2 * (2 if past else 1)
        elif kind == "delta":
            flops += 6 * B * L * m["heads"] * m["dim"] * m["vdim"]
            state += 4 * B * m["heads"] * m["dim"] * m["vdim"] * (2 if past else 1)
        elif kind == "rglru":
            state += 4 * B * W * (2 if past else 1)
        elif kind == "latent_attention":
            flops += 2 * B * seen * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            state += 2 * B * (past + L) * (m["kv_rank"] + m["rot_dim"])
        elif kind == "attention":
            flops += 4 * B * seen * m["heads"] * m["dim"]
            state += 2 * B * (past + L) * m["kv_heads"] * (m["dim"] + 2)
        else:
            flops += 4 * B * L * m["heads"] * m["dim"] * m["vdim"]
            state += 4 * B * m["heads"] * m["dim"] * m["vdim"] * (2 if past else 1)
    return {"bytes": 2 * (matrices + size[head]) + state + 8 * B * L + 2 * B * _vocab(cfg), "flops": flops}


def tolerance(case):
    if case["kind"] in ("prompt", "step"):
        return {"rel": 3e-2, "max": 0.5}     # 27 layers of bfloat16 activations; states of late layers differ most
    if case["kind"] == "mixer":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "decode" and case["state"] == "float32":
        return {"rel": 5e-3, "max": 5e-2}
    return {"rel": 1e-2, "max": 1e-1}


# --------------------------------------------------------------------------- exact results, in 64 bits

def _rms(x, w, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _linattn(q, k, v, eps=1e-12):
    """q, k ``[B, H, L, 16]``, v ``[B, H, L, dv]``: read-out and the two states, by chunks of the sequence."""
    B, H, L, _ = q.shape
    n, y = 512, torch.empty_like(v)
    S = torch.zeros(B, H, v.shape[-1], 273, dtype=v.dtype, device=v.device)
    z = torch.zeros(B, H, 273, dtype=v.dtype, device=v.device)
    for a in range(0, L, n):
        qc, kc, vc = q[:, :, a:a + n], k[:, :, a:a + n], v[:, :, a:a + n]
        x = qc @ kc.transpose(-1, -2) / 4
        p = (1 + x + x * x / 2).tril()
        fq, fk = _taylor(qc), _taylor(kc)
        y[:, :, a:a + n] = (p @ vc + fq @ S.transpose(-1, -2)) / (p.sum(-1, keepdim=True) + (fq * z[:, :, None]).sum(-1, keepdim=True) + eps)
        S += vc.transpose(-1, -2) @ fk
        z += fk.sum(2)
    return y, S.unsqueeze(2), z[:, :, None, None]


def _window(q, k, v, W):
    """q, k, v ``[B, L, H, d]``; query i sees keys i - W .. i."""
    q, k, v = (t.transpose(1, 2) for t in (q, k, v))
    L, n, out = q.shape[2], 512, torch.empty_like(v)
    for a in range(0, L, n):
        b, lo = min(a + n, L), max(0, a - W)
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(lo, b, device=q.device)[None]
        s = (q[:, :, a:b] @ k[:, :, lo:b].transpose(-1, -2)) * q.shape[-1] ** -0.5
        out[:, :, a:b] = s.masked_fill((j > i) | (j < i - W), -math.inf).softmax(-1) @ v[:, :, lo:b]
    return out.transpose(1, 2)


def _rotate(x, pos, base=1e4):
    """x ``[B, L, H, d]`` at positions ``pos [L]``; dimension i is paired with i + d / 2."""
    d = x.shape[-1]
    ang = pos.double()[:, None] * base ** (-2 * torch.arange(d // 2, device=x.device, dtype=torch.float64) / d)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    u, v = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, scale, past, sink=0.0):
    """q ``[B, L, H, d]`` at positions ``past ..``, k, v ``[B, T, H, d]``; ``sink`` scores of 0 in each softmax sum."""
    q, k, v = (t.transpose(1, 2) for t in (q, k, v))
    out, n = torch.empty(*q.shape[:3], v.shape[-1], dtype=q.dtype, device=q.device), 1024
    for a in range(0, q.shape[2], n):
        b = min(a + n, q.shape[2])
        T = past + b
        s = (q[:, :, a:b] @ k[:, :, :T].transpose(-1, -2)) * scale
        i, j = torch.arange(past + a, T, device=q.device)[:, None], torch.arange(T, device=q.device)[None]
        s = s.masked_fill(j > i, -math.inf)
        m = s.amax(-1, keepdim=True).clamp(min=0)
        e = torch.exp(s - m)
        out[:, :, a:b] = (e @ v[:, :, :T]) / (e.sum(-1, keepdim=True) + sink * torch.exp(-m))
    return out.transpose(1, 2)


def _ring_conv(x, taps, bias, ring, pos):
    """Causal convolution ``x [B, L, C]`` by ``taps [C, n]`` from position ``pos``; position p is in slot p mod n of ``ring``."""
    n, L = taps.shape[1], x.shape[1]
    slots = torch.arange(pos - n + 1, pos, device=x.device)
    before = ring[:, slots % n] if pos else torch.zeros_like(ring[:, :n - 1])
    full = torch.cat([before, x], 1)
    y = sum(full[:, j:j + L] * taps[:, j] for j in range(n))
    last = torch.arange(max(0, L - n), L, device=x.device)
    ring = ring.clone()
    ring[:, (pos + last) % n] = x[:, last]
    return (y if bias is None else y + bias), ring


def _delta(h, w, p, m, state, pos, eps):
    B, L, _ = h.shape
    H, d, dv = m["heads"], m["dim"], m["vdim"]
    taps = torch.cat([w(p + n + ".conv") for n in "qkv"])
    y, ring = _ring_conv(torch.cat([h @ w(p + n).T for n in "qkv"], -1), taps, None, state[0], pos)
    q, k, v = (t.unflatten(-1, (H, -1)) for t in _silu(y).split([H * d, H * d, H * dv], -1))
    q = q / torch.sqrt(q.square().sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(h @ w(p + "b").T)
    g = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(h @ w(p + "a").T + w(p + "dt_bias"), threshold=40))
    S = state[1] if pos else torch.zeros_like(state[1])
    o = torch.empty_like(v)
    for t in range(L):
        S = S * g[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * u[:, :, None]
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    o = _rms(o, w(p + "norm"), eps) * _silu((h @ w(p + "g").T).unflatten(-1, (H, dv)))
    return o.flatten(2) @ w(p + "o").T, [ring, S]


def _rglru(h, w, p, m, state, pos, eps):
    x, y = h @ w(p + "x").T + w(p + "x.b"), _gelu(h @ w(p + "y").T + w(p + "y.b"))
    u, ring = _ring_conv(x, w(p + "conv"), w(p + "conv.b"), state[0], pos)
    blocks = u.unflatten(-1, (m["blocks"], -1))
    r, i = (torch.sigmoid((torch.einsum("bon,xtbn->xtbo", w(p + n), blocks) + w(p + n + ".b")).flatten(2)) for n in ("ra", "ri"))
    a = torch.exp(-8 * r * torch.nn.functional.softplus(w(p + "lam")))
    add = torch.sqrt(1 - a * a) * i * u
    S = state[1] if pos else torch.zeros_like(state[1])
    for t in range(h.shape[1]):
        S = torch.addcmul(add[:, t], a[:, t], S)
        add[:, t] = S
    return (add * y) @ w(p + "o").T, [ring, S]


def _latent(h, w, p, m, cache, pos, eps):
    B, L, _ = h.shape
    H, d, rd, r = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    at = torch.arange(pos, pos + L, device=h.device)
    if m.get("kv_from") is None:
        z = h @ w(p + "dkv").T
        cache[:, pos:pos + L] = torch.cat([_rms(z[..., :r], w(p + "dkv.norm"), eps), _rotate(z[:, :, None, r:], at)[:, :, 0]], -1)
    q = (_rms(h @ w(p + "dq").T, w(p + "dq.norm"), eps) @ w(p + "uq").T).unflatten(-1, (H, d + rd))
    q = torch.cat([q[..., :d], _rotate(q[..., d:], at)], -1)
    T = pos + L
    c, kr = cache[:, :T, :r], cache[:, :T, None, r:]
    k = torch.cat([(c @ w(p + "uk").T).unflatten(-1, (H, d)), kr.expand(-1, -1, H, -1)], -1)
    o = _attend(q, k, (c @ w(p + "uv").T).unflatten(-1, (H, -1)), m["scale"], pos)
    o = o * torch.sigmoid(h @ w(p + "g").T)[..., None]
    return o.flatten(2) @ w(p + "o").T


def _grouped(x, w, p, m, state, pos, eps):
    B, L, _ = x.shape
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    keys, factor = state[0].clone(), state[1].clone()
    T = pos + L
    keys[:, pos:T] = x @ w(p + "k").T
    k = keys[:, :T].unflatten(-1, (G, d))
    factor[..., pos:T] = torch.rsqrt(k[:, pos:].square().mean(-1) + eps).transpose(1, 2)
    at = torch.arange(pos, T, device=x.device)
    temp = 1 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]) + 1).double()
    q = _rms((x @ w(p + "q").T).unflatten(-1, (H, d)), w(p + "q.norm"), eps) * temp[:, None, None]
    kn = k * factor[..., :T].transpose(1, 2)[..., None] * w(p + "k.norm")
    o = _attend(q, kn.repeat_interleave(H // G, 2), k.repeat_interleave(H // G, 2), m["scale"], pos, sink=1.0)
    return (o.flatten(2) * torch.sigmoid(x @ w(p + "g").T)) @ w(p + "o").T, [keys, factor]


def _lightning(x, w, p, m, state, pos, eps):
    B, L, _ = x.shape
    q, k, v = (_silu(x @ w(p + n).T).unflatten(-1, (m["heads"], -1)).transpose(1, 2) for n in "qkv")
    # the decay as the float32 that a layer holds
    a = torch.tensor(m["decay"], dtype=torch.float32).double().to(x.device)[:, None, None]
    S = state[0] if pos else torch.zeros_like(state[0])
    o, n = torch.empty_like(v), 256
    for t in range(0, L, n):
        qc, kc, vc = (y[:, :, t:t + n] for y in (q, k, v))
        i = torch.arange(qc.shape[2], device=x.device, dtype=torch.float64)
        D = (a ** (i[:, None] - i[None]).clamp(min=0)).tril()
        o[:, :, t:t + n] = (qc @ kc.transpose(-1, -2) * D) @ vc + (qc * a ** (i + 1)[:, None]) @ S
        S = a ** len(i) * S + (kc * a ** (len(i) - 1 - i)[:, None]).transpose(-1, -2) @ vc
    o = _rms(o.transpose(1, 2).flatten(2), w(p + "norm"), eps) * torch.sigmoid(x @ w(p + "g").T)
    return o @ w(p + "o").T, [S]


def _based_layer(kind, h, w, p, m, state, pos):
    B, L, W = h.shape
    if kind == "linattn":
        q, k, v = ((h @ w(p + f"proj_{n}.weight").T).unflatten(-1, (m["heads"], -1)).transpose(1, 2) for n in "qkv")
        if pos:
            fk = _taylor(k)
            S, z = state[0] + (v.unsqueeze(-1) * fk.unsqueeze(-2)), state[1] + fk.unsqueeze(-2)
            fq = _taylor(q).unsqueeze(-2)
            y = ((S * fq).sum(-1) / ((z * fq).sum(-1) + 1e-12))
        else:
            y, S, z = _linattn(q, k, v)
        return y.transpose(1, 2).flatten(2) @ w(p + "out_proj.weight").T, [S, z]
    if kind == "window":
        qkv = (h @ w(p + "Wqkv.weight").T).view(B, L, 3, m["heads"], m["dim"])
        at = torch.arange(pos, pos + L, device=h.device)
        cache = state[0].clone()
        cache[:, pos:pos + L, 0], cache[:, pos:pos + L, 1] = _rotate(qkv[:, :, 1], at), qkv[:, :, 2]
        lo = max(0, pos - 64)
        q = torch.zeros_like(cache[:, lo:pos + L, 0])
        q[:, pos - lo:] = _rotate(qkv[:, :, 0], at)
        o = _window(q, cache[:, lo:pos + L, 0], cache[:, lo:pos + L, 1], 64)[:, pos - lo:]
        return o.flatten(2) @ w(p + "out_proj.weight").T, [cache]
    u = h @ w(p + "in_proj.weight").T + w(p + "in_proj.bias")
    u1, u2 = u[..., :2 * W], u[..., 2 * W:]
    before = state[0].transpose(1, 2)[:, 1:] if pos else torch.zeros(B, KERNEL_SIZE - 1, 2 * W, dtype=h.dtype, device=h.device)
    full, taps = torch.cat([before, u1], 1), w(p + "conv.conv.weight")[:, 0]
    y = sum(full[:, j:j + L] * taps[:, j] for j in range(KERNEL_SIZE))
    tail = torch.cat([torch.zeros_like(full[:, :1]), full], 1)[:, -KERNEL_SIZE:]
    return (_silu(y) * u2) @ w(p + "out_proj.weight").T + w(p + "out_proj.bias"), [tail.transpose(1, 2)]


def _model(case, seed):
    cfg = _config(case["stack"])
    t = _weights(cfg, seed)
    w = lambda name: t[name].double()  # noqa: E731
    tokens, B, L, pos = _tokens(cfg, case, seed), case["B"], case.get("L", 1), case.get("pos", 0)
    if pos:
        states = [[s.double() for s in layer] for layer in _context(cfg, case, seed)]
    else:
        states = [[s.zero_().double() for s in layer] for layer in _context(cfg, dict(case, pos=1), seed)]
        for (kind, m, _, _), s in zip(_layers(cfg), states):   # caches of the prompt's own length
            if kind in ("window", "latent_attention", "attention") and s:
                shape = list(s[0].shape)
                shape[1] = L
                s[0] = torch.zeros(shape, dtype=torch.float64, device="cuda")
                if kind == "attention":
                    s[1] = torch.zeros(B, m["kv_heads"], (L + 127) // 128 * 128, dtype=torch.float64, device="cuda")
    out = []
    if cfg["architecture"] == "Based":
        x = w("transformer.embeddings.word_embeddings.weight")[tokens]
        for i, (kind, m, _, ff) in enumerate(_layers(cfg)):
            p = f"transformer.layers.{i}."
            y, s = _based_layer(kind, _rms(x, w(p + "norm1.weight"), 1e-5), w, p + "mixer.", m, states[i], pos)
            x = x + y
            u, gate = (_rms(x, w(p + "norm2.weight"), 1e-5) @ w(p + "mlp.fc1.weight").T).split(ff, -1)
            x = x + (u * _silu(gate)) @ w(p + "mlp.fc2.weight").T
            out.append(s)
        x = _rms(x[:, -1:], w("transformer.ln_f.weight"), 1e-5)
        return [x @ w("transformer.embeddings.word_embeddings.weight").T, out]
    eps = cfg["norm"]["eps"]
    mlp = lambda h, i: (_silu(h @ w(f"l{i}.mlp.gate").T) * (h @ w(f"l{i}.mlp.up").T)) @ w(f"l{i}.mlp.down").T  # noqa: E731
    if cfg["architecture"] == "Razesun":
        x = _rms(t["embed"][tokens].double(), w("embed.norm"), eps)
        for i, (kind, m, _, _) in enumerate(_layers(cfg)):
            h, p = _rms(x, w(f"l{i}.norm1"), eps), f"l{i}.mix."
            if kind == "latent_attention":
                src = m.get("kv_from")
                y, s = _latent(h, w, p, m, states[i if src is None else src][0], pos, eps), states[i]
            else:
                y, s = (_delta if kind == "delta" else _rglru)(h, w, p, m, states[i], pos, eps)
            x = x + cfg["residual_mult"] * (y + mlp(_rms(x, w(f"l{i}.norm2"), eps), i))
            out.append(s)
        return [_rms(x[:, -1:], w("final.norm"), eps) @ w("head").T, out]
    n = cfg["token_side"]["dim"]
    x = t["embed"][tokens].double() * cfg["embedding"]["scale"] + w("pos")[pos:pos + L]
    for i, (kind, m, _, _) in enumerate(_layers(cfg)):
        y, s = (_grouped if kind == "attention" else _lightning)(x, w, f"l{i}.mix.", m, states[i], pos, eps)
        x = x + _rms(y, w(f"l{i}.norm1"), eps)
        x = x + _rms(mlp(x, i), w(f"l{i}.norm2"), eps)
        side = t["side.embed"][:, i * n:(i + 1) * n][tokens].double()
        x = x + _rms((_gelu(x @ w(f"l{i}.side.gate").T) * side) @ w(f"l{i}.side.proj").T, w(f"l{i}.side.norm"), eps)
        out.append(s)
    return [_rms(x[:, -1:], w("final.norm"), eps) @ w("embed").T, out]


@torch.inference_mode()
def exact(case, seed):
    k = case["kind"]
    if k in ("prompt", "step"):
        return _model(case, seed)
    x = {n: t.double() if torch.is_tensor(t) else t for n, t in _inputs(case, seed).items()}
    if k == "decode":
        fk, fq = _taylor(x["k"])[:, :, None, None], _taylor(x["q"])[:, :, None, None]
        S, z = x["kv"] + x["v"][:, :, None, :, None] * fk, x["ks"] + fk
        y = (S * fq).sum(-1) / ((z * fq).sum(-1) + 1e-12)
        return [y.flatten(1).unsqueeze(1), S, z]
    if k == "linattn":
        parts = [_linattn(x["q"][b:b + 1], x["k"][b:b + 1], x["v"][b:b + 1]) for b in range(case["B"])]
        return [torch.cat(t) for t in zip(*parts)]
    if k == "window":
        return torch.cat([_window(*(t[:, :, j] for j in range(3)), case["window"]) for t in x["qkv"].split(1)])
    wq, wk, wv, wo = (t.double() for t in x["w"])
    q, kk, v = ((x["x"] @ t.T).unflatten(-1, (case["H"], -1)).transpose(1, 2) for t in (wq, wk, wv))
    y, S, z = _linattn(q, kk, v)
    return [y.transpose(1, 2).flatten(2) @ wo.T, S, z]
