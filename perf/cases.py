"""The work that users of this library have it do, as cases that can be timed and checked.

Every case goes through the Python package as a program would: a GPT-2 forward pass or decode step on a model that stays
loaded, the steps of a layered decoder (prompts, then one token per sequence), and the operators of one transformer block
called one by one.  Sizes are the repository's own (GPT-2 124M and XL; the layered decoders of its benchmark at widths 768
and 1600) over the batch sizes and lengths that serving meets.

`exact` restates each model in 64 bits with plain torch.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

VOCAB, PADDED_VOCAB, MAX_T = 50257, 50304, 1024
GPT2 = {"124m": {"layers": 12, "heads": 12, "width": 768}, "xl": {"layers": 48, "heads": 25, "width": 1600}}
_stream = None


# ---------------------------------------------------------------- cases
def listed():
    return [
        # a short prompt of one user: 64 tokens, latency, replayed as a graph
        {"name": "gpt2_forward_1x64", "kind": "forward", "model": "124m", "batch": 1, "length": 64, "mode": "bf16x3", "graph": True},
        # a ragged little batch
        {"name": "gpt2_forward_3x448", "kind": "forward", "model": "124m", "batch": 3, "length": 448, "mode": "bf16x3", "graph": False},
        # the benchmark's batch: scoring or evaluating long texts
        {"name": "gpt2_forward_8x1024", "kind": "forward", "model": "124m", "batch": 8, "length": 1024, "mode": "bf16x3", "graph": False},
        # the large model, the largest piece of work
        {"name": "gpt2_xl_forward_4x1024", "kind": "forward", "model": "xl", "batch": 4, "length": 1024, "mode": "bf16x3", "graph": False},
        # one user's next token behind a long text
        {"name": "gpt2_decode_1", "kind": "decode", "model": "124m", "batch": 1, "position": 897},
        # eight users' next tokens
        {"name": "gpt2_decode_8", "kind": "decode", "model": "124m", "batch": 8, "position": 543},
        # the same on the large model, the most rows that it takes
        {"name": "gpt2_xl_decode_8", "kind": "decode", "model": "xl", "batch": 8, "position": 300},
        # one transformer block from the operators, as a program with its own driver calls them
        {"name": "operators_8x1024", "kind": "operators", "width": 768, "heads": 12, "batch": 8, "length": 1024},
        # layered decoders: a step with prompts of unequal lengths ...
        {"name": "vunolorn_prompts", "kind": "layered", "design": "Vunolorn", "size": "1600", "layers": 8, "prompts": "1024,1,700,333,64,1019,511", "new": 0},
        {"name": "pumotar_prompts", "kind": "layered", "design": "Pumotar", "size": "768", "layers": 12, "prompts": "1024,1024,1024,1024,129,1024,1024,1024", "new": 0},
        # ... and a request's whole life: short prompts, then token by token
        {"name": "vunolorn_decode_3", "kind": "layered", "design": "Vunolorn", "size": "768", "layers": 12, "prompts": "37,250,101", "new": 16},
        {"name": "pumotar_decode_8", "kind": "layered", "design": "Pumotar", "size": "768", "layers": 12, "prompts": "64,3,97,41,128,77,19,50", "new": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "decode", "decode", "operators", "layered", "layered"])
    if kind == "forward":
        model = rng.choice(["124m", "124m", "xl"])
        length = 64 * rng.randint(1, 16)
        batch = min(_log_int(rng, 1, 8), 8 if model == "124m" else max(1, 4096 // length))
        return {"kind": kind, "model": model, "batch": batch, "length": length, "mode": rng.choice(["bf16x3", "bf16x3", "bf16x3", "tf32", "bf16"]),
                "graph": rng.random() < 0.5}
    if kind == "decode":
        model = rng.choice(["124m", "124m", "xl"])
        return {"kind": kind, "model": model, "batch": rng.randint(1, 16 if model == "124m" else 8), "position": rng.randint(0, MAX_T - 1)}
    if kind == "operators":
        heads = rng.choice([12, 16, 20, 25])
        return {"kind": kind, "width": 64 * heads, "heads": heads, "batch": _log_int(rng, 1, 8), "length": 64 * rng.randint(1, 16)}
    design, size = rng.choice(["Vunolorn", "Pumotar"]), rng.choice(["768", "1600"])
    layers = 4 * rng.randint(1, 3) if size == "768" else 4 if design == "Pumotar" else 8
    if rng.random() < 0.5:
        prompts = [_log_int(rng, 1, 1024) for _ in range(rng.randint(1, 8))]
        new = 0
    else:
        prompts = [_log_int(rng, 1, 256) for _ in range(rng.randint(1, 16))]
        new = rng.randint(4, 16)
    return {"kind": kind, "design": design, "size": size, "layers": layers, "prompts": ",".join(map(str, prompts)), "new": new}


# ---------------------------------------------------------------- inputs
def _package():
    path = os.path.join(os.getcwd(), "cuda-gpt2-inference_b200", "__init__.py")
    spec = importlib.util.spec_from_file_location("cuda_gpt2_inference_b200", path, submodule_search_locations=[os.path.dirname(path)])
    if spec.name not in sys.modules:
        sys.modules[spec.name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[spec.name])
    return sys.modules[spec.name]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


class _State:
    """What a program holds: a context on the program's stream, the model, inputs.  The device memory goes with it."""

    def __init__(self, pkg, case):
        global _stream
        if _stream is None:
            _stream = torch.cuda.Stream()
        self.case, self.ctx, self.model = case, pkg.Context(0, _stream), None

    def __del__(self):
        if self.model is not None:
            self.model.close()
        self.ctx.close()


def _gpt2_shapes(size):
    L, C = size["layers"], size["width"]
    return [("wte", (PADDED_VOCAB, C)), ("wpe", (MAX_T, C)), ("ln1w", (L, C)), ("ln1b", (L, C)), ("qkvw", (L, 3 * C, C)), ("qkvb", (L, 3 * C)),
            ("attprojw", (L, C, C)), ("attprojb", (L, C)), ("ln2w", (L, C)), ("ln2b", (L, C)), ("fcw", (L, 4 * C, C)), ("fcb", (L, 4 * C)),
            ("fcprojw", (L, C, 4 * C)), ("fcprojb", (L, C)), ("lnfw", (C,)), ("lnfb", (C,))]


def _gpt2_fill(size, flat, seed):
    """Parameters with the spreads of a trained model, in place; returns the tensors by name."""
    g, at, out = _generator(seed), 0, {}
    L, C = size["layers"], size["width"]
    for name, shape in _gpt2_shapes(size):
        n = math.prod(shape)
        t = flat[at:at + n].view(shape)
        at += n
        if name.startswith("ln") and name.endswith("w"):
            t.normal_(1.0, 0.1, generator=g)
        elif name.endswith("b"):
            t.normal_(0.0, 0.05, generator=g)
        elif name in ("wte", "wpe"):
            t.normal_(0.0, 0.1 if name == "wte" else 0.02, generator=g)
        else:
            t.normal_(0.0, 1.4 / math.sqrt(C if name != "fcprojw" else 4 * C) / (math.sqrt(2 * L) if "proj" in name else 1.0), generator=g)
        out[name] = t
    return out


def _gpt2_tokens(case, seed):
    n = case["length"] if case["kind"] == "forward" else MAX_T
    return torch.randint(0, VOCAB, (case["batch"], n), generator=_generator(seed + 1), device="cuda", dtype=torch.int32)


def _prompt_length(position):
    """The part of a text that is in the cache before the step: whole blocks of 64 by one prefill, the rest by steps."""
    return position // 64 * 64


SIZES = {
    "768": dict(width=768, heads=12, kv=4, ff=3072, inner=1536, rank=48, state=16, dh=12, dkv=6, dd=64, dv=128,
                rot=32, kv_rank=256, experts=16, top=2, eff=768, sff=1536),
    "1600": dict(width=1600, heads=25, kv=5, ff=6400, inner=3200, rank=100, state=16, dh=25, dkv=25, dd=128, dv=128,
                 rot=64, kv_rank=512, experts=16, top=2, eff=1600, sff=3200),
}


def _layered_config(case):
    s, layers = SIZES[case["size"]], []
    delta = {"conv": 4, "dim": s["dd"], "heads": s["dh"], "kv_heads": s["dkv"], "vdim": s["dv"]}
    if case["design"] == "Vunolorn":
        att = {"dim": 64, "heads": s["heads"], "kv_heads": s["kv"], "rot": {"base": 10000.0, "dims": 64}, "scale": 0.125, "vdim": 64}
        par = {"type": "parallel", "mixer": {"left": att, "left_scale": 1.0, "right": {"width": s["width"]}, "right_scale": 1.0},
               "mlp": {"kind": "dense", "ff": s["ff"]}}
        mamba = {"type": "mamba1", "mixer": {"conv": 4, "dt_rank": s["rank"], "inner": s["inner"], "state": s["state"]}, "mlp": None}
        layers = [[par, mamba, mamba, {"type": "delta", "mixer": delta, "mlp": None}][i % 4] for i in range(case["layers"])]
    else:
        lat = {"heads": s["heads"], "dim": 64, "rot_dim": s["rot"], "vdim": 64, "kv_rank": s["kv_rank"], "scale": (64 + s["rot"]) ** -0.5,
               "rot": {"base": 10000.0, "dims": s["rot"]}}
        moe = {"kind": "moe", "expert": {"ff": s["eff"], "limit": 7.0}, "router": {"experts": s["experts"], "top": s["top"]},
               "shared": {"ff": s["sff"], "limit": 7.0}}
        layers = [{"type": "latent_attention" if i % 4 == 3 else "channel_delta", "mixer": lat if i % 4 == 3 else delta,
                   "mlp": moe if i else {"kind": "dense", "ff": s["ff"]}} for i in range(case["layers"])]
    return {"architecture": case["design"], "vocab": PADDED_VOCAB, "width": s["width"], "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "layers": layers}


def _layered_shapes(cfg):
    C, V, post = cfg["width"], cfg["vocab"], cfg["architecture"] == "Vunolorn"
    s = {"embed": (V, C), "final.norm": (C,)}
    if post:
        s["head"] = (V, C)
    for i, layer in enumerate(cfg["layers"]):
        p, x, m, mlp = f"l{i}", f"l{i}.mix", layer["mixer"], layer["mlp"]
        s[p + ".norm1"] = (C,)
        if post:
            s[p + ".norm1b"] = (C,)
        if layer["type"] == "mamba1":
            n, r, st = m["inner"], m["dt_rank"], m["state"]
            s.update({x + ".in": (2 * n, C), x + ".conv": (n, m["conv"]), x + ".conv.b": (n,), x + ".x": (r + 2 * st, n), x + ".dt": (n, r),
                      x + ".dt.b": (n,), x + ".A_log": (n, st), x + ".D": (n,), x + ".o": (C, n)})
        elif "delta" in layer["type"]:
            H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for n, rows in (("q", G * D), ("k", G * D), ("v", H * Dv)):
                s[f"{x}.{n}"], s[f"{x}.{n}.conv"] = (rows, C), (rows, m["conv"])
            s.update({x + ".b": (H, C), x + ".A_log": (H,), x + ".norm": (Dv,), x + ".o": (C, H * Dv)})
            if layer["type"] == "delta":
                s.update({x + ".a": (H, C), x + ".dt_bias": (H,), x + ".g": (H * Dv, C)})
            else:
                s.update({x + ".a1": (D, C), x + ".a2": (H * D, D), x + ".dt_bias": (H * D,), x + ".g1": (Dv, C), x + ".g2": (H * Dv, Dv)})
        elif layer["type"] == "latent_attention":
            H, D, Dr, Dv, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            s.update({x + ".q": (H * (D + Dr), C), x + ".dkv": (R + Dr, C), x + ".dkv.norm": (R,), x + ".uk": (H * D, R), x + ".uv": (H * Dv, R),
                      x + ".o": (C, H * Dv)})
        else:
            a, W, l, r = m["left"], m["right"]["width"], x + ".left", x + ".right"
            H, G, D, Dv = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            s.update({l + ".q": (H * D, C), l + ".k": (G * D, C), l + ".v": (G * Dv, C), l + ".q.norm": (D,), l + ".k.norm": (D,), l + ".o": (C, H * Dv)})
            s.update({r + ".z": (W, C), r + ".z.b": (W,), r + ".x": (W, C), r + ".x.b": (W,), r + ".g": (W, C), r + ".o": (C, W)})
        if mlp is None:
            continue
        s[p + ".norm2"] = (C,)
        if post:
            s.update({p + ".norm2b": (C,), p + ".mlp.up": (mlp["ff"], C), p + ".mlp.down": (C, mlp["ff"])})
            continue
        parts = [(p + ".mlp", mlp["ff"])] if mlp["kind"] == "dense" else [(f"{p}.mlp.e{e}", mlp["expert"]["ff"]) for e in range(mlp["router"]["experts"])]
        if mlp["kind"] == "moe":
            parts.append((p + ".mlp.shared", mlp["shared"]["ff"]))
            s.update({p + ".mlp.table": (V, mlp["router"]["top"]), p + ".mlp.shared.sg": (1, C)})
        for q, F in parts:
            s.update({q + ".gate": (F, C), q + ".up": (F, C), q + ".down": (C, F)})
    return s


def _layered_weights(cfg, seed):
    """bf16 values (tables int32) on the GPU: activations of order one, slow and fast decays."""
    g, w = _generator(seed), {}
    for name, shape in _layered_shapes(cfg).items():
        leaf = name.rsplit(".", 1)[-1]
        if leaf == "table":
            experts = next(l["mlp"]["router"]["experts"] for l in cfg["layers"] if l["mlp"] and l["mlp"]["kind"] == "moe")
            w[name] = torch.rand((shape[0], experts), generator=g, device="cuda").argsort(dim=1)[:, :shape[1]].to(torch.int32).contiguous()
            continue
        t = torch.empty(shape, device="cuda")
        if leaf in ("norm1", "norm2") or name == "final.norm":
            t.normal_(0.0 if cfg["architecture"] == "Pumotar" else 1.0, 0.1, generator=g)
        elif "norm" in leaf or leaf == "D":
            t.normal_(1.0, 0.1, generator=g)
        elif leaf == "A_log":
            t.uniform_(-2.0, 1.5, generator=g)
        elif leaf == "dt_bias" or name.endswith(".dt.b"):
            t.uniform_(-5.0, -0.5, generator=g)
        elif leaf == "b" and len(shape) == 1:
            t.normal_(0.0, 0.5, generator=g)
        elif name == "embed":
            t.normal_(0.0, 0.2 if cfg["architecture"] == "Pumotar" else 1.0, generator=g)
        else:
            t.normal_(0.0, shape[-1] ** -0.5, generator=g)
        w[name] = t.to(torch.bfloat16)
    return w


def _layered_tokens(case, seed):
    """Per sequence: its prompt and the tokens that follow."""
    g = np.random.default_rng(seed + 1)
    return [g.integers(0, VOCAB, int(n) + case["new"]).astype(np.int32) for n in case["prompts"].split(",")]


def _operator_inputs(case, seed):
    g, C, M = _generator(seed), case["width"], case["batch"] * case["length"]
    n = lambda *s, std=1.0, mean=0.0: torch.empty(s, device="cuda").normal_(mean, std, generator=g)  # noqa: E731
    w = {"x": n(M, C)}
    for name, oc, c in (("qkv", 3 * C, C), ("proj", C, C), ("fc", 4 * C, C), ("fcproj", C, 4 * C)):
        w[name + ".w"], w[name + ".b"] = n(oc, c, std=1.4 / math.sqrt(c)), n(oc, std=0.05)
    for name in ("ln1", "ln2"):
        w[name + ".w"], w[name + ".b"] = n(C, std=0.1, mean=1.0), n(C, std=0.05)
    return w


def prepare(case, seed):
    pkg = _package()
    s = _State(pkg, case)
    if case["kind"] in ("forward", "decode"):
        size = GPT2[case["model"]]
        cfg = pkg.GPT2Config(num_layers=size["layers"], num_heads=size["heads"], channels=size["width"])
        s.model = pkg.GPT2(s.ctx, cfg, case["batch"], case["length"] if case["kind"] == "forward" else MAX_T)
        _gpt2_fill(size, s.model.params_tensor(), seed)
        s.tokens = _gpt2_tokens(case, seed)
        if case["kind"] == "forward":
            s.model.set_options(use_graph=int(case["graph"]), **pkg.MODES[case["mode"]])
        else:
            s.model.set_options(use_graph=1)
            s.model.enable_kv_cache()
            at = _prompt_length(case["position"])
            s.columns = s.tokens.t().contiguous()  # a step's tokens side by side
            prompt = s.tokens[:, :at].contiguous()
            torch.cuda.synchronize()
            if at:
                s.model.prefill(prompt, case["batch"], at)
            for t in range(at, case["position"]):
                s.model.decode_step(s.columns[t], case["batch"], t)
    elif case["kind"] == "layered":
        cfg = _layered_config(case)
        s.parts = _layered_tokens(case, seed)
        lens = [len(p) for p in s.parts]
        s.model = pkg.Decoder(s.ctx, cfg, "bfloat16", max_slots=len(lens), max_seq=max(lens), max_rows=max(64, min(8192, sum(lens))))
        s.model.load_tensors({k: (v if v.dtype == torch.int32 else v.view(torch.int16)).cpu().numpy().view(np.int32 if v.dtype == torch.int32 else np.uint16)
                              for k, v in _layered_weights(cfg, seed).items()})
        s.prompts = [p[:len(p) - case["new"]] for p in s.parts]
        s.steps = [[p[len(p) - case["new"] + i:][:1] for p in s.parts] for i in range(case["new"])]
    else:
        C, M = case["width"], case["batch"] * case["length"]
        s.w = _operator_inputs(case, seed)
        s.out = {k: torch.empty(M, n, device="cuda") for k, n in (("ln1", C), ("qkv", 3 * C), ("att", C), ("proj", C), ("res", C), ("ln2", C), ("fch", 4 * C),
                                                                  ("fcproj", C), ("out", C))}
        s.out["lse"] = torch.empty(case["batch"], case["heads"], case["length"], device="cuda")
        for k in ("mean1", "rstd1", "mean2", "rstd2"):
            s.out[k] = torch.empty(M, device="cuda")
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s.case
    if case["kind"] in ("forward", "decode"):
        if case["kind"] == "forward":
            logits = s.model.forward(s.tokens, case["batch"], case["length"])
        else:
            logits = s.model.decode_step(s.columns[case["position"]], case["batch"], case["position"])
        logits.owner = s  # a view of the model's buffer: the model stays while it is in use
        return logits
    if case["kind"] == "layered":
        slots = [s.model.open() for _ in s.prompts]
        out = [s.model.step(list(zip(slots, s.prompts)))]
        for tokens in s.steps:
            out.append(s.model.step(list(zip(slots, tokens))))
        for x in slots:
            s.model.close_slot(x)
        return out
    c, w, o = s.ctx, s.w, s.out
    B, T, C, NH = case["batch"], case["length"], case["width"], case["heads"]
    c.layernorm_forward(o["ln1"], o["mean1"], o["rstd1"], w["x"], w["ln1.w"], w["ln1.b"], B, T, C)
    c.matmul_forward(o["qkv"], o["ln1"], w["qkv.w"], w["qkv.b"], B, T, C, 3 * C)
    c.attention_forward(o["att"], None, o["lse"], o["qkv"], B, T, C, NH)
    c.matmul_forward(o["proj"], o["att"], w["proj.w"], w["proj.b"], B, T, C, C)
    c.fused_residual_layernorm_forward(o["res"], o["ln2"], o["mean2"], o["rstd2"], w["x"], o["proj"], w["ln2.w"], w["ln2.b"], B, T, C)
    c.matmul_forward(o["fch"], o["ln2"], w["fc.w"], w["fc.b"], B, T, C, 4 * C, act=1)
    c.matmul_forward(o["fcproj"], o["fch"], w["fcproj.w"], w["fcproj.b"], B, T, 4 * C, C)
    c.residual_forward(o["out"], o["res"], o["fcproj"], B * T * C)
    return o


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    if case["kind"] in ("forward", "decode"):
        size = GPT2[case["model"]]
        L, C = size["layers"], size["width"]
        matrices = L * 12 * C * C + PADDED_VOCAB * C
        if case["kind"] == "forward":
            M, T = case["batch"] * case["length"], case["length"]
            return {"bytes": 4.0 * matrices + 4.0 * M + 4.0 * M * PADDED_VOCAB, "flops": 2.0 * M * matrices + 2.0 * M * (T + 1) * C * L}
        B, n = case["batch"], case["position"] + 1
        return {"bytes": 4.0 * matrices + 8.0 * B * n * C * L + 4.0 * B * PADDED_VOCAB, "flops": 2.0 * B * matrices + 4.0 * B * n * C * L}
    if case["kind"] == "operators":
        C, M, T = case["width"], case["batch"] * case["length"], case["length"]
        return {"bytes": 4.0 * (12 * C * C + M * C * 15.0), "flops": 2.0 * M * 12 * C * C + 2.0 * M * (T + 1) * C}
    cfg, lens = _layered_config(case), [int(x) for x in case["prompts"].split(",")]
    dense = routed = active = attention = 0
    for name, shape in _layered_shapes(cfg).items():
        if len(shape) == 2 and not name.endswith((".table", ".conv", ".A_log")) and name != "embed":
            if ".mlp.e" in name:
                routed += math.prod(shape)
                active += math.prod(shape) * SIZES[case["size"]]["top"] / SIZES[case["size"]]["experts"]
            else:
                dense += math.prod(shape)
    head = PADDED_VOCAB * cfg["width"]
    layers = dense - (head if case["design"] == "Vunolorn" else 0)
    state = 0  # operations of a recurrence per token
    for l in cfg["layers"]:
        m = l["mixer"]
        if "delta" in l["type"]:
            state += 7 * m["heads"] * m["dim"] * m["vdim"]
        elif l["type"] == "mamba1":
            state += 6 * m["inner"] * m["state"]
        else:
            a = m.get("left", m)
            attention += 2 * a["heads"] * (a["dim"] + a.get("rot_dim", 0) + a["vdim"])
    B, new = len(lens), case["new"]
    touched = lambda rows: routed * (1 - (1 - SIZES[case["size"]]["top"] / SIZES[case["size"]]["experts"]) ** rows)  # noqa: E731
    tokens = sum(lens) + B * new
    pairs = sum((n + new) * (n + new + 1) / 2 for n in lens)
    nbytes = 2.0 * (layers + head + touched(sum(lens))) + new * 2.0 * (layers + head + touched(B)) + 4.0 * (1 + new) * B * PADDED_VOCAB
    return {"bytes": nbytes, "flops": tokens * (2.0 * (layers + active) + state) + 2.0 * (1 + new) * B * head + attention * pairs}


def tolerance(case):
    """Four times the distance from `exact` that the arithmetic of the path shows."""
    if case["kind"] == "forward":
        return {"rel": {"bf16x3": 1e-3, "tf32": 8e-3, "bf16": 4e-2}[case["mode"]]}
    if case["kind"] == "decode":  # the keys and values come from a prefill in the default arithmetic
        return {"rel": 8e-4}
    if case["kind"] == "operators":
        return {"rel": 2e-2}
    # (the norm behind the delta rule enlarges what rounding leaves of a sequence's first outputs where query and key hardly meet)
    return {"rel": 4e-2 if case["design"] == "Vunolorn" else 1.2e-1}


# ---------------------------------------------------------------- the same in 64 bits
def _layernorm(x, w, b):
    m = x.mean(-1, keepdim=True)
    v = ((x - m) ** 2).mean(-1, keepdim=True)
    return (x - m) / torch.sqrt(v + 1e-5) * w + b, m[..., 0], 1 / torch.sqrt(v[..., 0] + 1e-5)


def _gelu_tanh(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _attention(q, k, v, scale):
    """Causal attention of q [B,T,H,D], k [B,T,G,D], v [B,T,G,Dv]; also the log of the softmax sums [B,H,T]."""
    per, T = q.shape[2] // k.shape[2], q.shape[1]
    out, lse = torch.empty(*q.shape[:3], v.shape[3], dtype=q.dtype, device=q.device), []
    mask = torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1)
    for h in range(q.shape[2]):
        a = (q[:, :, h] @ k[:, :, h // per].transpose(1, 2) * scale).masked_fill(mask, -math.inf)
        out[:, :, h] = a.softmax(-1) @ v[:, :, h // per]
        lse.append(a.logsumexp(-1))
    return out, torch.stack(lse, 1)


def _gpt2_exact(size, flat, seed, tokens):
    w = _gpt2_fill(size, flat, seed)
    d = lambda name, l=None: (w[name] if l is None else w[name][l]).double()  # noqa: E731
    C, NH = size["width"], size["heads"]
    B, T = tokens.shape
    x = d("wte")[tokens.long()] + d("wpe")[:T]
    for l in range(size["layers"]):
        qkv = _layernorm(x, d("ln1w", l), d("ln1b", l))[0] @ d("qkvw", l).T + d("qkvb", l)
        q, k, v = qkv.view(B, T, 3, NH, 64).unbind(2)
        x = x + _attention(q, k, v, 0.125)[0].reshape(B, T, C) @ d("attprojw", l).T + d("attprojb", l)
        h = _gelu_tanh(_layernorm(x, d("ln2w", l), d("ln2b", l))[0] @ d("fcw", l).T + d("fcb", l))
        x = x + h @ d("fcprojw", l).T + d("fcprojb", l)
    return _layernorm(x, d("lnfw"), d("lnfb"))[0], d("wte")


def _rms(x, eps, w=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _conv(x, taps, bias=0.0):
    n, y = taps.shape[1], 0.0
    for j in range(n):
        back = n - 1 - j
        y = y + torch.nn.functional.pad(x, (0, 0, back, 0))[:, :x.shape[1]] * taps[:, j]
    return torch.nn.functional.silu(y + bias)


def _rotate(x, dims, base, pairs):
    """x [B,T,H,D]: the first `dims` dimensions turn; pairs (2i, 2i+1) or (i, i + dims/2)."""
    half = dims // 2
    a = torch.arange(x.shape[1], device=x.device).double()[:, None] * (float(base) ** (-2.0 * torch.arange(half, device=x.device).double() / dims))
    c, s = a.cos()[:, None], a.sin()[:, None]
    if pairs:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _mixer(kind, h, w, p, m, eps):
    B, T, _ = h.shape
    silu, softplus, sigmoid = torch.nn.functional.silu, lambda z: torch.logaddexp(z, torch.zeros_like(z)), torch.sigmoid
    if kind == "mamba1":
        n, r, st = m["inner"], m["dt_rank"], m["state"]
        x, z = (h @ w(p + ".in").T).split(n, -1)
        x = _conv(x, w(p + ".conv"), w(p + ".conv.b"))
        a, b, c = (x @ w(p + ".x").T).split([r, st, st], -1)
        dt = softplus(a @ w(p + ".dt").T + w(p + ".dt.b"))
        A, S, y = -torch.exp(w(p + ".A_log")), 0.0, torch.empty_like(x)
        for t in range(T):
            S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * x[:, t])[:, :, None] * b[:, t, None]
            y[:, t] = (S @ c[:, t, :, None])[..., 0]
        return ((y + w(p + ".D") * x) * silu(z)) @ w(p + ".o").T
    if "delta" in kind:
        H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_conv(h @ w(f"{p}.{n}").T, w(f"{p}.{n}.conv")) for n in "qkv")
        q, k = (_unit(x.view(B, T, G, D)).repeat_interleave(H // G, 2) for x in (q, k))
        q, v, beta = q * D ** -0.5, v.view(B, T, H, Dv), sigmoid(h @ w(p + ".b").T)
        rate = -torch.exp(w(p + ".A_log"))
        if kind == "delta":
            g = torch.exp(rate * softplus(h @ w(p + ".a").T + w(p + ".dt_bias")))[..., None].expand(B, T, H, D)
            gate = silu(h @ w(p + ".g").T)
        else:
            g = torch.exp(rate[:, None] * softplus(h @ w(p + ".a1").T @ w(p + ".a2").T + w(p + ".dt_bias")).view(B, T, H, D))
            gate = sigmoid(h @ w(p + ".g1").T @ w(p + ".g2").T)
        S, o = torch.zeros(B, H, D, Dv, dtype=h.dtype, device=h.device), torch.empty_like(v)
        for t in range(T):
            S = S * g[:, t, :, :, None]
            u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
            S = torch.addcmul(S, k[:, t, :, :, None], u[:, :, None])
            o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        return (_rms(o, eps, w(p + ".norm")) * gate.view(B, T, H, Dv)).reshape(B, T, H * Dv) @ w(p + ".o").T
    if kind == "latent_attention":
        H, D, Dr, Dv, R, base = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["rot"]["base"]
        q = (h @ w(p + ".q").T).view(B, T, H, D + Dr)
        q = torch.cat([q[..., :D], _rotate(q[..., D:], Dr, base, True)], -1)
        c, r = (h @ w(p + ".dkv").T).split([R, Dr], -1)
        c, r = _rms(c, eps, w(p + ".dkv.norm")), _rotate(r[:, :, None], Dr, base, True).expand(B, T, H, Dr)
        k = torch.cat([(c @ w(p + ".uk").T).view(B, T, H, D), r], -1)
        return _attention(q, k, (c @ w(p + ".uv").T).view(B, T, H, Dv), m["scale"])[0].reshape(B, T, H * Dv) @ w(p + ".o").T
    a, l, r = m["left"], p + ".left", p + ".right"
    H, G, D, Dv, rot = a["heads"], a["kv_heads"], a["dim"], a["vdim"], a["rot"]
    q = _rotate(_rms((h @ w(l + ".q").T).view(B, T, H, D), eps, w(l + ".q.norm")), rot["dims"], rot["base"], False)
    k = _rotate(_rms((h @ w(l + ".k").T).view(B, T, G, D), eps, w(l + ".k.norm")), rot["dims"], rot["base"], False)
    v = _rms((h @ w(l + ".v").T).view(B, T, G, Dv), eps)
    left = _attention(q, k, v, a["scale"])[0].reshape(B, T, H * Dv) @ w(l + ".o").T
    z, x = sigmoid(h @ w(r + ".z").T + w(r + ".z.b")), h @ w(r + ".x").T + w(r + ".x.b")
    x = z * torch.where(x >= 0, x + 0.5, sigmoid(x))
    S, y = 0.0, torch.empty_like(x)
    for t in range(T):
        S = (1 - z[:, t]) * S + x[:, t]
        y[:, t] = S
    return m["left_scale"] * left + m["right_scale"] * ((y * silu(h @ w(r + ".g").T)) @ w(r + ".o").T)


def _clamped(h, w, q, limit):
    g, u = (h @ w(q + ".gate").T).clamp(max=limit), (h @ w(q + ".up").T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(q + ".down").T


def _layered_exact(case, seed):
    cfg = _layered_config(case)
    weights, parts = _layered_weights(cfg, seed), _layered_tokens(case, seed)
    w = lambda name: weights[name].double()  # noqa: E731
    eps, post = cfg["norm"]["eps"], cfg["architecture"] == "Vunolorn"
    one = 0.0 if post else 1.0
    tokens = torch.zeros(len(parts), max(map(len, parts)), dtype=torch.long, device="cuda")  # what follows a sequence's end touches none of its outputs
    for i, t in enumerate(parts):
        tokens[i, :len(t)] = torch.from_numpy(t.astype(np.int64))
    x = w("embed")[tokens]
    for i, layer in enumerate(cfg["layers"]):
        p, mlp = f"l{i}", layer["mlp"]
        y = _mixer(layer["type"], _rms(x, eps, one + w(p + ".norm1")), w, p + ".mix", layer["mixer"], eps)
        x = x + (_rms(y, eps, w(p + ".norm1b")) if post else y)
        if mlp is None:
            continue
        h = _rms(x, eps, one + w(p + ".norm2"))
        if post:
            u = h @ w(p + ".mlp.up").T
            x = x + _rms((0.5 * u * (1 + torch.erf(u / math.sqrt(2)))) @ w(p + ".mlp.down").T, eps, w(p + ".norm2b"))
        elif mlp["kind"] == "dense":
            x = x + (_gelu_tanh(h @ w(p + ".mlp.gate").T) * (h @ w(p + ".mlp.up").T)) @ w(p + ".mlp.down").T
        else:
            flat, table, y = h.reshape(-1, h.shape[-1]), weights[p + ".mlp.table"][tokens.reshape(-1)], 0.0
            y = torch.sigmoid(flat @ w(p + ".mlp.shared.sg").T) * _clamped(flat, w, p + ".mlp.shared", mlp["shared"]["limit"])
            for e in range(mlp["router"]["experts"]):
                rows = (table == e).any(1).nonzero()[:, 0]
                y[rows] += _clamped(flat[rows], w, f"{p}.mlp.e{e}", mlp["expert"]["limit"]) / mlp["router"]["top"]
            x = x + y.view_as(h)
    x, head = _rms(x, eps, one + w("final.norm")), w("head" if post else "embed")
    rows = torch.arange(len(parts), device="cuda")
    ends = torch.tensor([len(t) for t in parts], device="cuda") - case["new"] - 1
    return [x[rows, ends + i] @ head.T for i in range(1 + case["new"])]


def exact(case, seed):
    if case["kind"] in ("forward", "decode"):
        size = GPT2[case["model"]]
        flat = torch.empty(sum(math.prod(s) for _, s in _gpt2_shapes(size)), device="cuda")
        tokens = _gpt2_tokens(case, seed)
        if case["kind"] == "forward":
            x, head = _gpt2_exact(size, flat, seed, tokens)
            return x @ head.T
        x, head = _gpt2_exact(size, flat, seed, tokens[:, :case["position"] + 1])
        return x[:, -1] @ head.T
    if case["kind"] == "layered":
        return _layered_exact(case, seed)
    w = {k: v.double() for k, v in _operator_inputs(case, seed).items()}
    B, T, C, NH = case["batch"], case["length"], case["width"], case["heads"]
    o = {}
    o["ln1"], o["mean1"], o["rstd1"] = _layernorm(w["x"], w["ln1.w"], w["ln1.b"])
    o["qkv"] = o["ln1"] @ w["qkv.w"].T + w["qkv.b"]
    att, o["lse"] = _attention(*o["qkv"].view(B, T, 3, NH, 64).unbind(2), 0.125)
    o["att"] = att.reshape(B * T, C)
    o["proj"] = o["att"] @ w["proj.w"].T + w["proj.b"]
    o["res"] = w["x"] + o["proj"]
    o["ln2"], o["mean2"], o["rstd2"] = _layernorm(o["res"], w["ln2.w"], w["ln2.b"])
    o["fch"] = _gelu_tanh(o["ln2"] @ w["fc.w"].T + w["fc.b"])
    o["fcproj"] = o["fch"] @ w["fcproj.w"].T + w["fcproj.b"]
    o["out"] = o["res"] + o["fcproj"]
    return o
