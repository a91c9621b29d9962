"""The framework's work as a user's program has it done, case by case, for measuring it.

A case is one call sequence through the public entry points, on a random-weight model of the table's or the
benchmark's sizes (`layers` cuts the depth; the matrices keep their full size):

  step     one decoded token at a KV context of `ctx` tokens (Engine.step), with or without the repetition penalty
           over the tokens so far: what a chat or a generation pays for each token
  prompt   `tokens` prompt tokens from position `pos0` on (Engine.prefill) and the step that yields the first answer
           token: the time to the first token of a request
  extend   a portion of a sequence through a model directory's design (Engine.extend) with the logits of some places
  reply    a short prompt and `steps` further tokens through a design with a recurrence, whose positions go in order

Weights and inputs come from generators with stated seeds.  The model file of a case is made once and kept in the
system's temporary memory, as a user keeps a checkpoint.
"""
from __future__ import annotations

import json
import math
import os
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

from cuqwen_b200 import binfmt, stackfmt
from cuqwen_b200 import engine as E

PENALTY, EPS = float(np.float16(1.1)), float(np.float16(1e-6))      # the table's models take both in fp16
THETA = 1e6

# Layer sizes of the designs that are read from a model directory, as in the benchmark's sweep over them.
STACKS = {
    "1.5b": dict(width=1536, vocab=32000, side=128, rank=64, latent=(12, 128, 64, 128, 768, 512, 1024, 13440),
                 parallel=(12, 2, 128, 128, 64, 24, 64, 6400), delta=(12, 6, 128, 128, 4, 8064)),
    "7b": dict(width=3584, vocab=32000, side=256, rank=64, latent=(28, 128, 64, 128, 1536, 512, 4096, 25600),
               parallel=(28, 4, 128, 128, 64, 56, 64, 12928), delta=(28, 14, 128, 128, 4, 16896)),
}
DEPTH = {"0.5b": 24, "1.5b": 8, "3b": 6, "7b": 4, "14b": 3}          # of drawn cases: what a model file of a second or two holds


def step(name, model, layers, quant, ctx, history=False):
    return dict(name=name, kind="step", model=model, layers=layers, quant=quant, ctx=ctx, history=history)


def prompt(name, model, layers, quant, tokens, pos0=0):
    return dict(name=name, kind="prompt", model=model, layers=layers, quant=quant, tokens=tokens, pos0=pos0)


def stack(name, kind, design, size, layers, tokens, steps=0):
    return dict(name=name, kind=kind, design=design, size=size, layers=layers, tokens=tokens, steps=steps)


def listed():
    return [
        step("step 0.5b int4", "0.5b", 24, "int4", 255),                          # a whole small model near the start of a chat: launches count
        step("step 0.5b fp16 penalty", "0.5b", 24, "fp16", 1777, True),           # unquantised, the penalty over everything seen so far
        step("step 7b int4 8k", "7b", 28, "int4", 8192),                          # the headline configuration, whole
        step("step 14b int8 32k", "14b", 6, "int8", 31999),                       # the largest matrices, a nearly full cache
        prompt("prompt 0.5b int8 61", "0.5b", 24, "int8", 61),                    # a one-line question
        prompt("prompt 7b int4 500", "7b", 8, "int4", 500),                       # an ordinary message
        prompt("prompt 3b fp16 3001+1000", "3b", 12, "fp16", 3001, 1000),         # a later message of a long chat, ragged against every tile
        prompt("prompt 14b int8 8191", "14b", 4, "int8", 8191),                   # a document
        stack("falivik 7b step", "step", "falivik", "7b", 4, 1500),               # latent attention: a token behind 1500 others
        stack("falivik 1.5b extend 1999", "extend", "falivik", "1.5b", 8, 1999),  # and a portion longer than its window
        stack("gipotar 1.5b reply", "reply", "gipotar", "1.5b", 8, 19, 16),       # recurrent mixers: a short prompt and its answer
        stack("gipotar 7b extend 2500", "extend", "gipotar", "7b", 4, 2500),      # and a long one, over the border of a portion
    ]


def spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 4 + ["prompt"] * 3 + ["falivik step", "falivik extend", "gipotar reply", "gipotar extend"])
    if kind in ("step", "prompt"):
        model = rng.choice(list(DEPTH))
        quant = rng.choice(["int4", "int4", "int8", "fp16"])
        if kind == "step":
            c = step("", model, DEPTH[model], quant, spread(rng, 1, 32000), rng.random() < 0.25)
        else:
            c = prompt("", model, DEPTH[model], quant, spread(rng, 2, 6000), rng.choice([0, 0, rng.randrange(1, 2000)]))
    else:
        design, kind = kind.split()
        size = rng.choice(list(STACKS))
        c = stack("", kind, design, size, 8 if size == "1.5b" else 4, spread(rng, 2, 3000 if kind == "extend" else 60 if kind == "reply" else 2000), spread(rng, 2, 24) if kind == "reply" else 0)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# model files
# ---------------------------------------------------------------------------
def is_table(case):
    return "model" in case


def model_place(case) -> Path:
    what = "%s_%s_%d" % ((case["model"], case["quant"], case["layers"]) if is_table(case) else (case["design"], case["size"], case["layers"]))
    base = Path("/dev/shm") if os.access("/dev/shm", os.W_OK) and shutil.disk_usage("/dev/shm").free > 48 << 30 else Path(tempfile.gettempdir())
    return base / f"cuqwen_case_{os.getuid()}_{what}"


def table_config(case):
    return dict(binfmt.MODELS[case["model"]], layers=case["layers"])


def file_order(cfg):
    """(name, rows or 0 for a vector, columns, whether it is quantised) of a model file's tensors, in its order."""
    d, q, k, i, v = cfg["dim"], cfg["heads"] * cfg["hd"], cfg["kv"] * cfg["hd"], cfg["inter"], cfg["vocab"]
    yield "embed", v, d, False
    for n in range(cfg["layers"]):
        yield f"{n}.norm1", 0, d, False
        for s, rows in (("q", q), ("k", k), ("v", k)):
            yield f"{n}.{s}", rows, d, True
            yield f"{n}.b{s}", 0, rows, False
        yield f"{n}.o", d, q, True
        yield f"{n}.norm2", 0, d, False
        yield f"{n}.gate", i, d, True
        yield f"{n}.up", i, d, True
        yield f"{n}.down", d, i, True
    yield "norm", 0, d, False
    if not cfg["tied"]:
        yield "head", v, d, True


def quant_of(name, quant):
    return "int8" if name == "head" and quant != "fp16" else quant


def write_table_model(path, cfg, quant):
    """Weights ~ N(0, 0.02) (norms about one), quantised in groups of 128 columns as the exporter does."""
    gen = torch.Generator("cuda").manual_seed(42)
    fmt = binfmt.lm_head_fmt(binfmt.QUANT_ID[quant], cfg["tied"])
    with open(path, "wb") as f:
        f.write(binfmt.Header(cfg["vocab"], cfg["dim"], cfg["inter"], cfg["layers"], cfg["heads"], cfg["kv"], cfg["hd"], 32768, binfmt.QUANT_ID[quant], fmt).pack())
        for name, rows, cols, packed in file_order(cfg):
            w = torch.randn((rows or 1, cols), generator=gen, device="cuda") * 0.02 + (1.0 if "norm" in name else 0.0)
            kind = quant_of(name, quant) if packed else "fp16"
            if kind == "fp16":
                w.half().cpu().numpy().tofile(f)
                continue
            top = 7 if kind == "int4" else 127
            g = w.view(rows, -1, 128)
            s = g.abs().amax(2) / top
            v = (g / s[..., None]).round_().clamp_(-top, top).to(torch.int8).view(rows, cols)
            if kind == "int4":
                v = (v[:, 0::2] & 15) | (v[:, 1::2] << 4)
            v.cpu().numpy().tofile(f)
            s.half().cpu().numpy().tofile(f)


def stack_config(case):
    z = STACKS[case["size"]]
    if case["design"] == "falivik":                     # the last layer of four attends to the latents of the one before
        ls = [stackfmt.latent_layer(*z["latent"], kv_from=i - 1 if i % 4 == 3 else None) for i in range(case["layers"])]
        return stackfmt.falivik_config(z["vocab"], z["width"], z["side"], ls)
    return stackfmt.gipotar_config(z["vocab"], z["width"], [stackfmt.parallel_layer(*z["parallel"]) if i % 2 else stackfmt.delta_layer(*z["delta"]) for i in range(case["layers"])],
                                   residual_mult=0.4)


def model_file(case) -> Path:
    """The case's checkpoint, made when it is not there yet."""
    p = model_place(case)
    if not p.exists():
        tmp = p.with_name(p.name + ".%d" % os.getpid())
        if is_table(case):
            write_table_model(tmp, table_config(case), case["quant"])
        else:
            cfg = stack_config(case)
            stackfmt.write_model_dir(tmp, cfg, stackfmt.random_weights(cfg, 42, block=1 << 20, rank=STACKS[case["size"]]["rank"]))
        os.replace(tmp, p)
    return p


# ---------------------------------------------------------------------------
# state and call
# ---------------------------------------------------------------------------
class View:
    """Engine memory as torch sees it; keeps the engine while a tensor of it lives."""

    def __init__(self, eng, which, shape, typestr):
        self.eng = eng
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (eng.ptr(which)[0], False), "version": 3}

    def tensor(self):
        return torch.as_tensor(self, device="cuda")


def random_tokens(case, seed, n):
    vocab = table_config(case)["vocab"] if is_table(case) else STACKS[case["size"]]["vocab"]
    return np.random.default_rng([seed, 1]).integers(0, vocab, size=n).astype(np.int32)


def fill_rows(cfg, seed, rows):
    """Random keys and values of `rows` cached tokens, layer by layer: N(0, 1) in fp16."""
    gen = torch.Generator("cuda").manual_seed(seed)
    for _ in range(cfg["layers"]):
        yield tuple(torch.randn((cfg["kv"], rows, cfg["hd"]), generator=gen, device="cuda").half() for _ in range(2))


def prepare(case, seed):
    path, kind = model_file(case), case["kind"]
    if not is_table(case):
        eng = E.Engine.open(path)
        vocab = STACKS[case["size"]]["vocab"]
        toks = random_tokens(case, seed, case["tokens"] + case["steps"] + (kind == "step"))
        if kind == "step":
            eng.prefill(toks[:-1], 0)
        return dict(kind=kind, eng=eng, toks=toks, n=case["tokens"], want=wanted(case), logits=View(eng, "LOGITS", (vocab,), "<f4").tensor())
    cfg = table_config(case)
    prm = E.model_params(case["model"], case["quant"])
    if case["layers"] != binfmt.MODELS[case["model"]]["layers"]:
        prm = E.custom_params(cfg["vocab"], cfg["dim"], cfg["inter"], cfg["layers"], cfg["heads"], cfg["kv"], cfg["hd"], case["quant"])
    eng = E.Engine(prm)
    eng.load(str(path))
    shape = (cfg["layers"], cfg["kv"], eng.params.max_seq_len, cfg["hd"])
    cache = [View(eng, s, shape, "<f2").tensor() for s in ("KEY_CACHE", "VALUE_CACHE")]
    first, n = (case["ctx"], 1) if kind == "step" else (case["pos0"], case["tokens"])
    if first:
        for i, kv in enumerate(fill_rows(cfg, seed, first)):
            for c, new in zip(cache, kv):
                c[i, :, :first] = new
    toks = random_tokens(case, seed, first + n)
    out = {"logits": View(eng, "LOGITS", (cfg["vocab"],), "<f2").tensor(), "keys": cache[0][:, :, first:first + n], "values": cache[1][:, :, first:first + n]}
    return dict(kind=kind, eng=eng, toks=toks[first:], pos=first, history=toks if case.get("history") else None, out=out)


def run(s):
    eng, toks = s["eng"], s["toks"]
    if "out" in s:
        n, pos = len(toks), s["pos"]
        if n > 1:
            eng.prefill(toks[:-1], pos)
        eng.step(int(toks[-1]), pos + n - 1, s["history"])
        return s["out"]
    n = s["n"]
    if s["kind"] == "step":
        eng.step(int(toks[n]), n)
        return s["logits"]
    out = {"prompt": eng.extend(toks[:n], 0, s["want"])}
    if s["kind"] == "reply":
        for i in range(n, len(toks)):
            eng.step(int(toks[i]), i)
        out["reply"] = s["logits"]
    return out


def wanted(case):
    """Places whose logits a portion returns: its last one, and for a long one some before it."""
    n = case["tokens"]
    return [n - 1] if case["kind"] == "reply" else sorted({n - 1} | {n * i // 8 for i in range(1, 8)})


# ---------------------------------------------------------------------------
# bytes and operations that a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    if is_table(case):
        cfg, q = table_config(case), binfmt.QUANT_ID[case["quant"]]
        first, n = (case["ctx"], 1) if case["kind"] == "step" else (case["pos0"], case["tokens"])
        d, qd, kd = cfg["dim"], cfg["heads"] * cfg["hd"], cfg["kv"] * cfg["hd"]
        layer = d * (2 * qd + 2 * kd + 3 * cfg["inter"])
        keys = n * first + n * (n + 1) // 2
        # the last layer of all tokens but the last ends with their keys and values
        flops = 2 * n * cfg["layers"] * layer - 2 * (n - 1) * (layer - 2 * d * kd) + 2 * d * cfg["vocab"] + 4 * qd * (keys * (cfg["layers"] - 1) + first + n)
        kv_rows = 2 * cfg["layers"] * kd * 2
        return {"bytes": binfmt.step_bytes(cfg, q, first) + kv_rows * n + (n - 1) * d * 2 + cfg["vocab"] * 2, "flops": flops}
    cfg = stack_config(case)
    shapes = (stackfmt.falivik_shapes if case["design"] == "falivik" else lambda c: stackfmt.gipotar_shapes(c, STACKS[case["size"]]["rank"]))(cfg)
    n = 1 if case["kind"] == "step" else case["tokens"] + case["steps"]
    weights = sum(math.prod(s) for k, s in shapes.items() if "embed" not in k and k != "head")
    matrices = sum(math.prod(s) for k, s in shapes.items() if "embed" not in k and k != "head" and len(s) == 2 and "conv" not in k)
    head = math.prod(shapes["head"])
    n_logits = len(wanted(case)) + case["steps"] if case["kind"] != "step" else 1
    mix = keys_bytes = 0
    for L in cfg["layers"]:
        m = L["mixer"]
        if L["type"] == "latent_attention":
            w, first = m["mask"]["size"], case["tokens"] if case["kind"] == "step" else 0
            pairs = sum(min(first + i + 1, w) for i in range(n))
            mix += 2 * pairs * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            keys_bytes += 2 * min(first, w) * (m["kv_rank"] + m["rot_dim"])
        elif L["type"] == "parallel":
            a, t = m["left"], m["right"]
            mix += n * (n + 1) * a["heads"] * (a["dim"] + a["vdim"]) + 6 * n * t["heads"] * t["dim"] ** 2
        else:
            mix += 8 * n * m["heads"] * m["dim"] * m["vdim"]
    passes = 1 + case["steps"]                              # a token that waits for the one before reads the weights again
    return {"bytes": passes * 2 * (weights + head) + keys_bytes + 2 * n * cfg["width"] + 4 * n_logits * cfg["vocab"],
            "flops": 2 * n * matrices + 2 * n_logits * head + mix}


def tolerance(case):
    """fp16 or bfloat16 activations between float32 sums, over the layers of a model: about four times the error against
    64 bits that was measured (0.002 to 0.005).  Random logits are nearly flat, so values are compared and not the token."""
    return {"rel": 0.015 if is_table(case) else 0.02, "max": 0.15}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
F64 = torch.float64


def rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def rotate(x, pos, base, dims):
    """The first `dims` entries of x [n, heads, d], entry i with entry i + dims / 2."""
    half = dims // 2
    ang = pos.to(F64)[:, None] * torch.pow(torch.tensor(float(base), dtype=F64, device="cuda"), -2.0 * torch.arange(half, device="cuda", dtype=F64) / dims)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def attend(q, k, v, scale, first, window=0, sink=None):
    """q [n, H, d] at positions first .., k and v [m, G, .] from position 0 on, causal; `sink`: one more term of a head's denominator."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=F64, device="cuda")
    own = torch.arange(k.shape[0], device="cuda")
    for a in range(0, n, 512):
        b = min(n, a + 512)
        at = torch.arange(first + a, first + b, device="cuda")[:, None]
        seen = (own <= at) & ((own > at - window) if window else True)
        for h in range(H):
            s = (q[a:b, h] @ k[:, h * G // H].T * scale).masked_fill_(~seen, -math.inf)
            z = s if sink is None else torch.cat([s, sink[h].expand(b - a, 1)], 1)
            out[a:b, h] = torch.softmax(z, 1)[:, :k.shape[0]] @ v[:, h * G // H]
    return out


def read_table_model(case):
    """name -> its weights in 64 bits, read from the model file when asked for."""
    cfg, raw, off, place = table_config(case), np.memmap(model_file(case), np.uint8, "r"), 256, {}
    for name, rows, cols, packed in file_order(cfg):
        kind = quant_of(name, case["quant"]) if packed else "fp16"
        nb = (rows or 1) * cols * {"fp16": 4, "int8": 2, "int4": 1}[kind] // 2
        place[name] = (kind, rows, cols, off, nb)
        off += nb + (0 if kind == "fp16" else rows * cols // 128 * 2)

    def get(name, some=None):
        kind, rows, cols, at, nb = place[name]
        data = raw[at:at + nb].view(np.float16 if kind == "fp16" else np.int8)
        if kind == "fp16":
            data = data.reshape(rows, cols)[some] if some is not None else data.reshape(rows, cols) if rows else data
            return torch.from_numpy(np.array(data)).cuda().to(F64)
        q = torch.from_numpy(np.array(data)).cuda()
        if kind == "int4":
            q = torch.stack([(q << 4) >> 4, q >> 4], 1)
        s = torch.from_numpy(np.array(raw[at + nb:at + nb + rows * cols // 128 * 2].view(np.float16))).cuda().to(F64)
        return (q.reshape(-1, 128).to(F64) * s[:, None]).view(rows, cols)

    return get


def exact_table(case, seed):
    cfg, get = table_config(case), read_table_model(case)
    first, n = (case["ctx"], 1) if case["kind"] == "step" else (case["pos0"], case["tokens"])
    toks = random_tokens(case, seed, first + n)
    H, G, hd = cfg["heads"], cfg["kv"], cfg["hd"]
    pos = torch.arange(first, first + n, device="cuda")
    x = get("embed", toks[first:])
    filled = fill_rows(cfg, seed, first) if first else None
    keys, values = [], []
    for i in range(cfg["layers"]):
        h = rms(x, get(f"{i}.norm1"), EPS)
        q, k, v = ((h @ get(f"{i}.{s}").T + get(f"{i}.b{s}")).view(n, -1, hd) for s in "qkv")
        q, k = rotate(q, pos, THETA, hd), rotate(k, pos, THETA, hd)
        keys.append(k.transpose(0, 1).contiguous())
        values.append(v.transpose(0, 1).contiguous())
        if first:
            k, v = (torch.cat([old.transpose(0, 1).to(F64), new]) for old, new in zip(next(filled), (k, v)))
        if i + 1 == cfg["layers"]:                         # only the last token goes on from here
            x, q = x[-1:], q[-1:]
        x = x + attend(q, k, v, hd ** -0.5, first + n - len(q)).reshape(len(q), -1) @ get(f"{i}.o").T
        h = rms(x, get(f"{i}.norm2"), EPS)
        x = x + (torch.nn.functional.silu(h @ get(f"{i}.gate").T) * (h @ get(f"{i}.up").T)) @ get(f"{i}.down").T
    logits = (rms(x, get("norm"), EPS) @ get("embed" if cfg["tied"] else "head").T)[0]
    if case.get("history"):
        seen = torch.from_numpy(np.unique(toks[:4096]).astype(np.int64)).cuda()
        z = logits[seen]
        logits[seen] = torch.where(z > 0, z / PENALTY, z * PENALTY)
    return {"logits": logits, "keys": torch.stack(keys), "values": torch.stack(values)}


def read_model_dir(path):
    raw = np.memmap(path / "model.safetensors", np.uint8, "r")
    n = int.from_bytes(bytes(raw[:8]), "little")
    head = json.loads(bytes(raw[8:8 + n]))

    def get(name, some=None):
        a, b = head[name]["data_offsets"]
        bits = raw[8 + n + a:8 + n + b].view(np.int16).reshape(head[name]["shape"])
        return torch.from_numpy(np.array(bits if some is None else bits[some])).cuda().view(torch.bfloat16).to(F64)

    return get


def falivik_layer(x, get, p, L, cfg, toks, pos, at, latents):
    m, eps, n = L["mixer"], cfg["norm"]["eps"], len(x)
    h1, q_ = rms(x, get(p + "norm1"), eps), p + "mix."
    if m.get("kv_from") is None:
        kv = h1 @ get(q_ + "dkv").T
        latents[at] = rms(kv[:, :m["kv_rank"]], get(q_ + "dkv.norm"), eps), rotate(kv[:, None, m["kv_rank"]:], pos, m["rot"]["base"], m["rot"]["dims"])
    c, kr = latents[at if m.get("kv_from") is None else m["kv_from"]]
    H, d = m["heads"], m["dim"]
    q = (rms(h1 @ get(q_ + "dq").T, get(q_ + "dq.norm"), eps) @ get(q_ + "uq").T).view(n, H, -1)
    q = torch.cat([q[..., :d], rotate(q[..., d:], pos, m["rot"]["base"], m["rot"]["dims"])], -1)
    k = torch.cat([(c @ get(q_ + "uk").T).view(n, H, d), kr.expand(n, H, -1)], -1)
    o = attend(q, k, (c @ get(q_ + "uv").T).view(n, H, -1), m["scale"], 0, m["mask"]["size"], get(q_ + "sink"))
    y = x + (o.reshape(n, -1) * torch.sigmoid(h1 @ get(q_ + "g").T)) @ get(q_ + "o").T
    if L["mlp"] is not None:
        y = y + torch.relu(rms(x, get(p + "norm2"), eps) @ get(p + "mlp.up").T).square() @ get(p + "mlp.down").T
    sd = cfg["token_side"]["dim"]
    e = get("side.embed", toks)[:, at * sd:(at + 1) * sd]
    return y + rms((torch.nn.functional.gelu(y @ get(p + "side.gate").T, approximate="tanh") * e) @ get(p + "side.proj").T, get(p + "side.norm"), eps)


def delta_mixer(h, get, p, m, eps):
    n, H, G, vd = len(h), m["heads"], m["kv_heads"], m["vdim"]
    parts = []
    for s in "qkv":
        z, taps = h @ get(p + s).T, get(f"{p}{s}.conv")
        z = torch.cat([z.new_zeros(taps.shape[1] - 1, z.shape[1]), z])
        parts.append(torch.nn.functional.silu(sum(z[i:i + n] * taps[:, i] for i in range(taps.shape[1]))))
    q, k = (z.view(n, G, -1) for z in parts[:2])
    q, k = (z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6) for z in (q, k))
    q, k = q.repeat_interleave(H // G, 1) * m["dim"] ** -0.5, k.repeat_interleave(H // G, 1)
    v, beta = parts[2].view(n, H, vd), torch.sigmoid(h @ get(p + "b").T)
    g = torch.exp(-torch.exp(get(p + "A_log")) * torch.nn.functional.softplus(h @ get(p + "a").T + get(p + "dt_bias")))
    S, o = q.new_zeros(H, m["dim"], vd), torch.empty_like(v)
    for t in range(n):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    o = rms(o, get(p + "norm"), eps) * torch.nn.functional.silu(h @ get(p + "g").T).view(n, H, vd)
    return o.reshape(n, -1) @ get(p + "o").T


def parallel_mixer(h, get, p, m, eps, pos):
    a, t, n = m["left"], m["right"], len(h)
    q, k, v = ((h @ get(f"{p}left.{s}").T).view(n, -1, a["vdim"] if s == "v" else a["dim"]) for s in "qkv")
    q, k = (rotate(z, pos, a["rot"]["base"], a["rot"]["dims"]) for z in (q, k))
    left = attend(q, k, v, a["scale"], 0).reshape(n, -1) @ get(p + "left.o").T
    p, before = p + "right.", torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    x = {s: h + (before - h) * get(f"{p}mu.{s}") for s in "rkvgw"}
    r, k, v = ((x[s] @ get(p + s).T).view(n, t["heads"], -1) for s in "rkv")
    w = torch.exp(-torch.exp(torch.tanh(x["w"] @ get(p + "w1").T) @ get(p + "w2").T + get(p + "w0"))).view(r.shape)
    u, S, o = get(p + "u"), r.new_zeros(t["heads"], t["dim"], t["dim"]), torch.empty_like(v)
    for i in range(n):
        kv = torch.bmm(k[i][:, :, None], v[i][:, None])
        o[i] = torch.bmm(r[i][:, None], torch.addcmul(S, u[:, :, None], kv))[:, 0]
        S = torch.addcmul(kv, w[i][:, :, None], S)
    o = rms(o, 1.0, eps).reshape(n, -1) * get(p + "norm")
    right = (o * torch.nn.functional.silu(x["g"] @ get(p + "g").T)) @ get(p + "o").T
    return m["left_scale"] * left + m["right_scale"] * right


def gipotar_layer(x, get, p, L, cfg, pos):
    eps, m = cfg["norm"]["eps"], L["mixer"]
    h = rms(x, 1.0 + get(p + "norm1"), eps)
    x = x + cfg["residual_mult"] * (parallel_mixer(h, get, p + "mix.", m, eps, pos) if L["type"] == "parallel" else delta_mixer(h, get, p + "mix.", m, eps))
    if L["mlp"] is not None:
        h, top = rms(x, 1.0 + get(p + "norm2"), eps), L["mlp"]["limit"]
        g, u = (h @ get(p + "mlp.gate").T).clamp(max=top), (h @ get(p + "mlp.up").T).clamp(-top, top)
        x = x + cfg["residual_mult"] * (g * torch.sigmoid(1.702 * g) * (u + 1)) @ get(p + "mlp.down").T
    return x


def exact_stack(case, seed):
    path = model_file(case)
    cfg, get = stack_config(case), read_model_dir(path)
    toks = random_tokens(case, seed, case["tokens"] + case["steps"] + (case["kind"] == "step"))
    pos, latents, gipotar = torch.arange(len(toks), device="cuda"), {}, case["design"] == "gipotar"
    x = get("embed", toks) * (cfg["embedding"]["scale"] if gipotar else 1.0)
    for i, L in enumerate(cfg["layers"]):
        x = gipotar_layer(x, get, f"l{i}.", L, cfg, pos) if gipotar else falivik_layer(x, get, f"l{i}.", L, cfg, toks, pos, i, latents)
    want = wanted(case) if case["kind"] != "step" else []
    x = x[want + ([len(toks) - 1] if case["kind"] != "extend" else [])]
    z = rms(x, get("final.norm") + (1.0 if gipotar else 0.0), cfg["norm"]["eps"]) @ get("head").T
    if gipotar:
        z = cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])
    return z[0] if case["kind"] == "step" else {"prompt": z[:-1], "reply": z[-1]} if case["kind"] == "reply" else {"prompt": z}


def exact(case, seed):
    with torch.no_grad():
        return exact_table(case, seed) if is_table(case) else exact_stack(case, seed)
