"""The framework's work as its users have it do, as cases that can be timed and compared.

Three architectures, each through its public entry points (ainfer_b200.runtime): prompts
(Session.prefill, prefill_logits), decoding of one sequence (Session.step, generate, sample), and
batches of sequences (BatchDecode). The INT4 hybrid runs the presets of the library; Sinepel and
Robopel models are folders with config.json and SafeTensors weights, at the widths, heads and
feed-forwards of the throughput table of `bench.py --design`.

The INT4 hybrid computes on quantised activations: every product is of whole numbers and every
32-bit sum has a stated order, so its outputs are compared bit for bit and have no 64-bit form.
"""
import json
import math
import os
import shutil
import struct
import tempfile
import weakref
import zlib

import numpy as np
import torch

from ainfer_b200 import cuda_abi, runtime

VOCAB = 32000
POSITIONS = 8192          # learned positions of a Sinepel model
STREAMS, TAPS = 4, 4
POOL = 16                 # tokens of a block mean (Robopel)
EPS = 1e-6

# The sizes of the INT4 hybrid's presets that a pass's work depends on.
PRESETS = {
    "mini": dict(layers="LA", hidden=1024, vocab=32000, q=8, kv=2, lk=8, lv=16, experts=64, top=4, ff=256),
    "small": dict(layers="LLLA", hidden=2048, vocab=32000, q=16, kv=2, lk=16, lv=32, experts=512, top=10, ff=512),
    "full": dict(layers="LLLA" * 12, hidden=2048, vocab=151936, q=16, kv=2, lk=16, lv=32, experts=512, top=10, ff=512),
}


# ------------------------------------------------------------------- the cases ---
def rows_model(arch, width, heads, kv_heads, ff, layers, span, dim=128, experts=0, identity=0, top=0, expert_ff=0):
    """A Sinepel (span: its chunk) or Robopel (span: its window) model's sizes, as plain values."""
    m = {"arch": arch, "width": width, "heads": heads, "kv_heads": kv_heads, "dim": dim, "ff": ff, "layers": layers, "span": span}
    if arch == "robopel":
        m.update(experts=experts, identity=identity, top=top, expert_ff=expert_ff)
    return m


SINEPEL_1024 = rows_model("sinepel", 1024, 8, 2, 4096, 2, 1024)
SINEPEL_2048 = rows_model("sinepel", 2048, 16, 4, 8192, 4, 2048)
ROBOPEL_1024 = rows_model("robopel", 1024, 8, 2, 4096, 2, 512, experts=16, identity=2, top=2, expert_ff=1024)
ROBOPEL_2048 = rows_model("robopel", 2048, 16, 4, 8192, 4, 1024, experts=32, identity=2, top=4, expert_ff=1024)


def listed():
    return [
        # a chat on the smallest preset: a step, then a draw from its logits, eight times; launches and latency
        {"name": "hybrid-chat-mini", "kind": "chat", "arch": "hybrid", "preset": "mini", "context": 100, "tokens": 8},
        # the 80B-shaped model answering one user at a 4096-token context: greedy tokens, batch 1
        {"name": "hybrid-decode-full", "kind": "generate", "arch": "hybrid", "preset": "full", "context": 4096, "tokens": 16},
        # the same model reading a prompt of ordinary, uneven length, up to its first token
        {"name": "hybrid-prompt-full", "kind": "prompt", "arch": "hybrid", "preset": "full", "tokens": 701},
        # the same model serving many users: one step of a batch
        {"name": "hybrid-batch-full", "kind": "batch", "arch": "hybrid", "preset": "full", "batch": 64, "context": 2048},
        # a long document into a bf16 model (two passes of rows)
        {"name": "sinepel-prompt", "kind": "prompt", **SINEPEL_2048, "tokens": 4096, "wanted": 1, "f32": False},
        # one user's continuation, token by token, late in a chunk
        {"name": "sinepel-decode", "kind": "steps", **SINEPEL_2048, "context": 1500, "tokens": 8, "f32": False},
        # a few users at once
        {"name": "sinepel-batch", "kind": "batch", **SINEPEL_2048, "batch": 16, "context": 600, "f32": False},
        # everything in 32-bit (--dtype float32): a prompt of uneven length
        {"name": "sinepel-prompt-f32", "kind": "prompt", **SINEPEL_1024, "tokens": 777, "wanted": 1, "f32": True},
        # scoring: the logits of the last 16 tokens of an uneven long text, mixtures and recurrences on the way
        {"name": "robopel-prompt", "kind": "prompt", **ROBOPEL_2048, "tokens": 3001, "wanted": 16, "f32": False},
        # a short question
        {"name": "robopel-prompt-short", "kind": "prompt", **ROBOPEL_1024, "tokens": 130, "wanted": 1, "f32": False},
        # one user's continuation on a small model: latency
        {"name": "robopel-decode", "kind": "steps", **ROBOPEL_1024, "context": 500, "tokens": 8, "f32": False},
        # many users at once
        {"name": "robopel-batch", "kind": "batch", **ROBOPEL_2048, "batch": 64, "context": 700, "f32": False},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    what = rng.choice(("hybrid", "hybrid", "hybrid", "sinepel", "sinepel", "sinepel", "robopel", "robopel", "robopel"))
    if what == "hybrid":
        kind, preset = rng.choice(("chat", "generate", "prompt", "batch")), rng.choice(("mini", "small", "full"))
        c = {"kind": kind, "arch": "hybrid", "preset": preset}
        if kind == "chat":
            return {**c, "context": _log_int(rng, 2, 1000), "tokens": rng.randint(4, 12)}
        if kind == "generate":
            return {**c, "context": _log_int(rng, 64, 4200), "tokens": rng.randint(4, 16)}
        if kind == "prompt":
            return {**c, "tokens": _log_int(rng, 5, 700 if preset == "full" else 2000)}
        return {**c, "batch": _log_int(rng, 2, 64), "context": _log_int(rng, 64, 2048)}
    # models between the two sizes of the list, heads of 64, 96 or 128
    dim, kv = rng.choice((64, 96, 128, 128)), rng.choice((1, 2, 4))
    heads = kv * rng.choice((2, 4, 4, 8)) if kv < 4 else kv * rng.choice((2, 4))
    m = rows_model(what, 8 * _log_int(rng, 96, 256), heads, kv, 8 * _log_int(rng, 256, 1024), rng.choice((2, 3, 4)), _log_int(rng, 200, 2048), dim,
                   experts=rng.choice((8, 16, 24, 32)), identity=rng.choice((0, 1, 2)), top=rng.choice((2, 3, 4)), expert_ff=8 * _log_int(rng, 48, 128))
    kind, f32 = rng.choice(("prompt", "prompt", "steps", "batch")), rng.random() < 0.15
    if kind == "prompt":
        tokens = _log_int(rng, 20, 800 if f32 else 4000)
        return {"kind": kind, **m, "tokens": tokens, "wanted": min(16, tokens) if what == "robopel" else 1, "f32": f32}
    if kind == "steps":
        return {"kind": kind, **m, "context": _log_int(rng, 30, 3000), "tokens": rng.randint(4, 12), "f32": f32}
    return {"kind": kind, **m, "batch": _log_int(rng, 2, 64), "context": _log_int(rng, 30, 700), "f32": f32}


# ------------------------------------------------------------- weights of rows ---
def _config(c):
    W, H, G, D, F = c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"]
    if c["arch"] == "sinepel":
        layer = {"type": "attention", "mlp": {"ff": F, "kind": "dense"},
                 "mixer": {"conv": TAPS, "dim": D, "heads": H, "kv_heads": G, "mask": {"size": c["span"]}, "scale": D ** -0.5, "vdim": D}}
        return {"architecture": "Sinepel", "embedding": {"scale": 1.0}, "layers": [layer] * c["layers"], "logit_softcap": 30.0,
                "max_positions": POSITIONS, "norm": {"eps": EPS}, "streams": STREAMS, "vocab": VOCAB, "width": W}
    layers = []
    for i in range(c["layers"]):
        if i % 2:
            layers.append({"type": "mingru", "mixer": {"width": W}, "mlp": {
                "expert": {"ff": c["expert_ff"]}, "kind": "moe", "router": {"experts": c["experts"], "identity": c["identity"], "top": c["top"]}}})
            continue
        m = {"dim": D, "heads": H, "kv_heads": G, "mask": {"pool": POOL, "size": c["span"]}, "scale": D ** -0.5, "softcap": 30.0, "vdim": D,
             "rot": {"base": 10000.0, "dims": D, "scaling": {"factor": 8.0, "high": 4.0, "low": 1.0, "original": 2048}}}
        if i:
            m["kv_from"] = 0
        layers.append({"type": "attention", "mixer": m, "mlp": {"ff": F, "kind": "dense"}})
    return {"architecture": "Robopel", "embedding": {"scale": 1.0}, "layers": layers, "norm": {"eps": EPS}, "vocab": VOCAB, "width": W}


def _shapes(c):
    """Every tensor of the model with its shape."""
    W, H, G, D, F = c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"]
    sh = {"embed": (VOCAB, W), "final.norm": (W,), "head": (VOCAB, W)}
    if c["arch"] == "sinepel":
        sh["pos"] = (POSITIONS, W)
    for i in range(c["layers"]):
        p = "l%d." % i
        x, f = p + "mix.", p + "mlp."
        sh.update({p + "norm1": (W,), p + "norm2": (W,)})
        if c["arch"] == "sinepel":
            sh.update({p + "shift": (W,), x + "q": (H * D, W), x + "q.b": (H * D,), x + "k": (G * D, W), x + "k.b": (G * D,),
                       x + "q.conv": (H * D, TAPS), x + "k.conv": (G * D, TAPS), x + "r1": (H,), x + "r2": (H,), x + "temp": (H,),
                       x + "o": (W, H * D), f + "up": (F, W), f + "down": (W, F)})
            for q in ("hc1.", "hc2."):
                sh.update({p + q + "in": (STREAMS,), p + q + "out": (STREAMS,), p + q + "mix": (STREAMS, STREAMS)})
        elif i % 2:
            n, E = c["experts"] + c["identity"], c["expert_ff"]
            sh.update({x + "z": (W, W), x + "x": (W, W), x + "g": (W, W), x + "z.b": (W,), x + "x.b": (W,), x + "o": (W, W), f + "router": (n, W),
                       f + "correction": (n,)})
            for e in range(c["experts"]):
                sh.update({f + "e%d.up" % e: (E, W), f + "e%d.down" % e: (W, E)})
        else:
            sh.update({x + "q": (H * D, W), x + "q.norm": (D,), x + "sink": (H,), x + "g": (H * D, W), x + "o": (W, H * D), f + "up": (F, W),
                       f + "down": (W, F), f + "act": (4,)})
            if not i:
                sh.update({x + "k": (G * D, W), x + "v": (G * D, W), x + "k.norm": (D,)})
    return sh


def _weights(c):
    """The model's bf16 weights on the GPU: matrices of unit gain, and every small tensor away from its neutral
    value. They depend on the sizes alone: a user opens one model and runs many inputs through it."""
    text = json.dumps(_config(c), sort_keys=True)
    g = torch.Generator("cuda").manual_seed(zlib.crc32(text.encode()))
    out = {}
    for n, s in sorted(_shapes(c).items()):
        r = torch.randn(s, generator=g, device="cuda")
        leaf = n.split(".", 1)[-1]
        if leaf in ("norm1", "norm2", "norm"):
            v = (1.0 if c["arch"] == "sinepel" else 0.0) + 0.2 * r
        elif leaf == "shift":
            v = torch.sigmoid(r)
        elif leaf == "mix.z.b":
            v = -2.0 + r
        elif leaf.endswith(".b"):
            v = 0.3 * r
        elif leaf.endswith(".conv"):
            v = 0.3 * r
            v[:, -1] += 0.8
        elif leaf in ("mix.r1", "mix.r2"):
            v = 0.2 + torch.sigmoid(r)
        elif leaf == "mix.temp":
            v = 0.6 + torch.sigmoid(r)
        elif leaf.startswith("hc"):
            v = 0.25 + 0.2 * r if leaf.endswith(".in") else 0.7 + 0.3 * r if leaf.endswith(".out") else 0.8 * torch.eye(s[0], device="cuda") + 0.15 * r
        elif leaf == "mix.q.norm":
            v = 1.5 + 0.2 * r
        elif leaf == "mix.k.norm":
            v = 1.0 + 0.2 * r
        elif leaf == "mix.sink":
            v = 1.0 + r
        elif leaf == "mlp.act":
            v = torch.tensor([0.7, -0.5, 0.4, 0.3], device="cuda") + 0.1 * r
        elif leaf == "mlp.router":
            v = 4.0 * r / math.sqrt(s[1])
        elif leaf == "mlp.correction":
            v = 0.01 * r
        elif n in ("embed", "pos"):
            v = 0.5 * r
        else:
            v = r / math.sqrt(s[1])
        out[n] = v.to(torch.bfloat16)
    return out


def _write_folder(folder, c):
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(_config(c), f)
    w = _weights(c)
    head, off = {}, 0
    for n in sorted(w):
        size = w[n].numel() * 2
        head[n] = {"dtype": "BF16", "shape": list(w[n].shape), "data_offsets": [off, off + size]}
        off += size
    text = json.dumps(head).encode()
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(text)) + text)
        for n in sorted(w):
            w[n].contiguous().view(torch.int16).cpu().numpy().tofile(f)


# -------------------------------------------------------------- states of a run ---
class _Model:
    """An open model, closed when the last state that uses it is gone."""

    def __init__(self, c):
        self.dev = cuda_abi.Device(0)
        if c["arch"] == "hybrid":
            self.model = runtime.Model(self.dev, "synth:%s:seed=0" % c["preset"])
        else:
            folder = tempfile.mkdtemp(dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
            try:
                _write_folder(folder, c)
                torch.cuda.empty_cache()
                self.model = runtime.Model(self.dev, folder)
            finally:
                shutil.rmtree(folder, ignore_errors=True)

    def __del__(self):
        if hasattr(self, "model"):
            self.model.close()
            self.dev.close()


_open = weakref.WeakValueDictionary()
_MODEL_KEYS = ("arch", "preset", "width", "heads", "kv_heads", "dim", "ff", "layers", "span", "experts", "identity", "top", "expert_ff")


def _model(c):
    key = tuple(c.get(k) for k in _MODEL_KEYS)
    m = _open.get(key)
    if m is None:
        m = _open[key] = _Model(c)
    return m


class _DeviceArray:
    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner       # the buffer lives as long as its views
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 3, "strides": None}


class _Owner:
    """A session or batch and its model, closed when neither a state nor a view of its buffers needs it any more."""

    def __init__(self, handle, m):
        self.handle, self.m = handle, m

    def view(self, which, kind, dtype_size, shape=None):
        """A torch view of one of the framework's device buffers."""
        ptr, size = self.handle.buffer(which)
        return torch.as_tensor(_DeviceArray(self, ptr, shape or (size // dtype_size,), kind), device="cuda")

    def __del__(self):
        self.handle.close()


class _State:
    def __init__(self, c, seed):
        self.c, m = c, _model(c)
        self.model = m.model
        rng = np.random.default_rng(seed)
        vocab, kind = self.model.config["vocab"], c["kind"]
        f32 = 32 if c.get("f32") else 0
        if kind == "batch":
            B, ctx = c["batch"], c["context"]
            self.handle = b = runtime.BatchDecode(self.model, B, ctx + 16, flags=f32)
            self.owner = _Owner(b, m)
            self.ids = rng.integers(0, vocab, (ctx + 1, B)).astype(np.int32)
            self.at = np.full(B, ctx, np.int32)
            if c["arch"] == "hybrid":
                self.fill(seed)
            else:
                for i in range(ctx):
                    b.set_inputs(self.ids[i], np.full(B, i, np.int32))
                    b.step()
            self.logits = self.owner.view("logits", "<f4", 4, (B, vocab))
            return
        total = c["tokens"] + c.get("context", 0)
        flags = f32 | (runtime.Session.PERSISTENT if c["arch"] == "hybrid" else 0)
        self.handle = s = runtime.Session(self.model, total + 24, flags)
        self.owner = _Owner(s, m)
        s.reset()
        self.ids = rng.integers(0, vocab, total).astype(np.int32)
        self.wanted = np.arange(c["tokens"] - c.get("wanted", 1), c["tokens"], dtype=np.int32)
        s.prefill(self.ids[:2])          # what a first call sets up
        s.reset()
        ctx = c.get("context", 0)
        if kind == "generate":
            self.fill(seed)
        elif ctx:
            s.prefill(self.ids[:ctx])
        self.logits = self.owner.view("logits", "<f4", 4, (vocab,))

    def fill(self, seed):
        """A hybrid's state late in a conversation: recurrent state, convolution history and INT8 cache."""
        g = torch.Generator("cuda").manual_seed(int(seed))
        for n in ("Kc", "Vc"):
            self.owner.view(n, "|i1", 1).random_(-127, 128, generator=g)
        for n in ("Ks", "Vs"):
            v = self.owner.view(n, "<f2", 2)
            v.copy_(0.008 + 0.008 * torch.rand(v.shape, generator=g, device="cuda"))
        self.owner.view("S", "<f4", 4).normal_(0, 0.1, generator=g)
        self.owner.view("conv", "<f4", 4).normal_(0, 1, generator=g)
        torch.cuda.synchronize()


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    c, h, ids = state.c, state.handle, state.ids
    kind = c["kind"]
    if kind == "batch":
        h.set_inputs(ids[-1], state.at)
        h.step()
        return {"logits": state.logits}
    if kind == "generate":
        tokens = h.generate(ids[c["context"]:c["context"] + 1], c["tokens"], start_pos=c["context"])
        return {"tokens": tokens, "logits": state.logits}
    if kind == "chat":
        tok, pos, draw_state, out = int(ids[c["context"]]), c["context"], 1234567, []
        for i in range(c["tokens"]):
            h.step(tok, pos + i)
            tok, draw_state = h.sample(0.8, 40, 0.95, rng=draw_state)
            out.append(tok)
        return {"tokens": np.array(out), "logits": state.logits}
    if kind == "steps":                     # given tokens: a continuation that is scored, or drawn elsewhere
        for i in range(c["context"], c["context"] + c["tokens"]):
            h.step(int(ids[i]), i)
        return {"logits": state.logits}
    if c["arch"] == "hybrid":
        h.reset()
        h.prefill(ids[:-1])
        tokens = h.generate(ids[-1:], 1, start_pos=len(ids) - 1)
        return {"tokens": tokens, "logits": state.logits}
    return {"logits": h.prefill_logits(ids, state.wanted)}


# --------------------------------------------------------------- work of a pass ---
def _rows(c):
    """(token rows of a pass, how often the weights cross memory, positions before the first row of a sequence, sequences, rows of logits)"""
    k = c["kind"]
    if k == "batch":
        return c["batch"], 1, c["context"], c["batch"], c["batch"]
    if k == "prompt":
        return c["tokens"], 1, 0, 1, c.get("wanted", 1)
    return c["tokens"], c["tokens"], c["context"], 1, c["tokens"]


def _touched(experts, choices, top, rows):
    """Experts that `rows` uniform choices of `top` out of `choices` touch."""
    return experts * (1 - (1 - top / choices) ** rows)


def _hybrid_work(c):
    p = PRESETS[c["preset"]]
    rows, times, before, seqs, heads = _rows(c)
    per = rows // times                       # rows that share one crossing of the weights
    w, H, D = 0.5 + 2.0 / 128, p["hidden"], 256
    lin, att = p["layers"].count("L"), p["layers"].count("A")
    cd, vd = (2 * p["lk"] + p["lv"]) * 128, p["lv"] * 128
    dense = lin * (cd * H + vd * H + 2 * p["lv"] * H + H * vd) + att * (p["q"] * 2 * D * H + 2 * p["kv"] * D * H + H * p["q"] * D)
    expert, n = 3 * p["ff"] * H, lin + att
    router = (p["experts"] + 1) * H
    state = lin * p["lv"] * 128 * 128 * 4 * 2 * (seqs if c["kind"] != "prompt" else 1) * times
    reach = before if c["kind"] != "prompt" else rows / 2
    kv = att * 2 * p["kv"] * (D + 2) * ((before + times / 2) * seqs * times if c["kind"] != "prompt" else rows)
    touched = _touched(p["experts"], p["experts"], p["top"], per) + 1
    b = times * (w * (dense + n * touched * expert + p["vocab"] * H) + 2 * n * router) + state + kv + heads * p["vocab"] * 4
    f = 2 * rows * (dense + n * ((p["top"] + 1) * expert + router)) + 2 * heads * p["vocab"] * H
    f += rows * (lin * p["lv"] * 128 * 128 * 8 + att * 4 * p["q"] * D * reach)
    return {"bytes": float(b), "flops": float(f)}


def _reach(c, first, rows):
    """Mean number of keys that rows first .. first + rows - 1 of a sequence meet in an attention layer."""
    i = np.arange(first, first + rows)
    if c["arch"] == "sinepel":
        return float((i % c["span"] + 1).mean())
    return float((np.minimum(i + 1, c["span"]) + np.maximum(0, i - c["span"] + 1) // POOL).mean())


def work(case):
    c = case
    if c["arch"] == "hybrid":
        return _hybrid_work(c)
    rows, times, before, seqs, heads = _rows(c)
    per, W, HD, GD = rows // times, c["width"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
    n = rows // seqs
    if c["arch"] == "sinepel":
        weights = active = c["layers"] * ((HD + GD) * W + HD * W + 2 * c["ff"] * W)
        attn, copies = c["layers"], 1
    else:
        attn, rec, copies = (c["layers"] + 1) // 2, c["layers"] // 2, 2
        choices = c["experts"] + c["identity"]
        dense = attn * (3 * HD * W + 2 * c["ff"] * W) + 2 * GD * W + rec * (4 * W * W + choices * W)
        one = 2 * c["expert_ff"] * W
        weights = dense + rec * _touched(c["experts"], choices, c["top"], per) * one
        active = dense + rec * c["top"] * c["experts"] / choices * one
    reach = _reach(c, before, n)
    esz = 4 if c["f32"] else 2
    keys = attn * copies * GD * esz * (rows if c["kind"] == "prompt" else rows * reach)
    b = times * 2 * (weights + VOCAB * W) + keys + heads * VOCAB * 4 + rows * W * 2
    f = 2 * rows * active + 2 * heads * VOCAB * W + rows * attn * 4 * HD * reach
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    if case["arch"] == "hybrid":
        return "exact"
    if case["f32"]:
        return {"rel": 1e-5}
    return {"rel": 0.02}


# --------------------------------------------------------------- in 64 bits ---
def _rms(x, gain=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if gain is None else y * gain


def _short_conv(u, taps):
    y, J = torch.zeros_like(u), taps.shape[1]
    for j in range(J):
        back = J - 1 - j
        y[back:] += u[:len(u) - back] * taps[:, j]
    return y


def _softmax_attention(q, k, v, scores):
    """q [T][H][D], k and v [n][G][D] -> [T][H][D]; scores(h, raw) gives the masked scores of a head."""
    T, H, _ = q.shape
    out, rep = torch.empty_like(q), H // k.shape[1]
    for h in range(H):
        s = scores(h, q[:, h] @ k[:, h // rep].T)
        out[:, h] = torch.softmax(s, -1)[:, :len(k)] @ v[:, h // rep]
    return out


class _Plain:
    """The two designs of rows as plain 64-bit torch, whole sequences at a time."""

    def __init__(self, c):
        self.c, self.w = c, _weights(c)

    def __call__(self, tokens, wanted):
        t = torch.as_tensor(tokens, dtype=torch.long, device="cuda")
        return (self.sinepel if self.c["arch"] == "sinepel" else self.robopel)(t, wanted)

    def d(self, name):
        return self.w[name].double()

    def sinepel(self, t, wanted):
        c, T, d = self.c, len(t), self.d
        H, G, D = c["heads"], c["kv_heads"], c["dim"]
        x = (self.w["embed"][t].double() + self.w["pos"][:T].double())[:, None, :].repeat(1, STREAMS, 1)
        i = torch.arange(T, device="cuda")
        far = (i[:, None] - i[None, :]).clamp(min=0).double()
        hidden = ~((i[:, None] >= i[None, :]) & (i[:, None] // c["span"] == i[None, :] // c["span"]))
        for n in range(c["layers"]):
            p = "l%d." % n

            def mixer(h):
                h = h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * d(p + "shift")
                q = _short_conv(h @ d(p + "mix.q").T + d(p + "mix.q.b"), d(p + "mix.q.conv")).reshape(T, H, D)
                k = _short_conv(h @ d(p + "mix.k").T + d(p + "mix.k.b"), d(p + "mix.k.conv")).reshape(T, G, D)
                temp, r1, r2 = d(p + "mix.temp"), d(p + "mix.r1"), d(p + "mix.r2")

                def scores(h, s):
                    return (s * (D ** -0.5) * temp[h] - r1[h] * torch.log1p(r2[h] * far)).masked_fill(hidden, -math.inf)
                return _softmax_attention(q, k, k, scores).reshape(T, H * D) @ d(p + "mix.o").T

            def ff(h):
                return torch.relu(h @ d(p + "mlp.up").T).square() @ d(p + "mlp.down").T
            for q, norm, f in (("hc1.", "norm1", mixer), ("hc2.", "norm2", ff)):
                h = _rms(torch.einsum("tsw,s->tw", x, d(p + q + "in")), d(p + norm))
                x = torch.einsum("tsw,su->tuw", x, d(p + q + "mix")) + d(p + q + "out")[None, :, None] * f(h)[:, None, :]
        return 30.0 * torch.tanh(_rms(x.sum(1)[wanted], d("final.norm")) @ d("head").T / 30.0)

    def rotate(self, x):
        D = x.shape[-1]
        a = []
        for i in range(D // 2):
            f = 10000.0 ** (-2.0 * i / D)
            wave = 2 * math.pi / f
            if wave > 2048:
                f /= 8.0
            elif wave >= 512:
                s = (2048 / wave - 1.0) / 3.0
                f = (1 - s) * f / 8.0 + s * f
            a.append(f)
        a = torch.arange(len(x), device="cuda").double()[:, None] * torch.tensor(a, dtype=torch.float64, device="cuda")
        a = a[:, None, :]
        u, v, y = x[..., 0::2], x[..., 1::2], torch.empty_like(x)
        y[..., 0::2], y[..., 1::2] = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
        return y

    def robopel(self, t, wanted):
        c, T, d = self.c, len(t), self.d
        H, G, D, S = c["heads"], c["kv_heads"], c["dim"], c["span"]
        x = self.w["embed"][t].double()
        i = torch.arange(T, device="cuda")
        back = i[:, None] - i[None, :]
        blocks = torch.arange(T // POOL, device="cuda")
        hidden = torch.cat([(back < 0) | (back >= S), (blocks[None, :] * POOL + POOL - 1) > (i[:, None] - S)], 1)
        kv = None
        for n in range(c["layers"]):
            p, h = "l%d." % n, x
            m = p + "mix."
            if n % 2:
                z, u = torch.sigmoid(h @ d(m + "z").T + d(m + "z.b")), h @ d(m + "x").T + d(m + "x.b")
                cand = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
                keep, gain, rows, s = 1 - z, z * cand, torch.empty_like(z), torch.zeros_like(z[0])
                for k in range(T):
                    s = torch.addcmul(gain[k], keep[k], s)
                    rows[k] = s
                g = h @ d(m + "g").T
                y = (rows * (g * torch.sigmoid(g))) @ d(m + "o").T
            else:
                q = self.rotate(_rms((h @ d(m + "q").T).reshape(T, H, D), d(m + "q.norm")))
                if not n:
                    k = self.rotate(_rms((h @ d(m + "k").T).reshape(T, G, D), d(m + "k.norm")))
                    v = (h @ d(m + "v").T).reshape(T, G, D)
                    whole = T // POOL * POOL
                    kv = [torch.cat([e, e[:whole].reshape(-1, POOL, G, D).mean(1)]) for e in (k, v)]
                sink = d(m + "sink")

                def scores(h, s):
                    s = (30.0 * torch.tanh(s * (D ** -0.5) / 30.0)).masked_fill(hidden, -math.inf)
                    return torch.cat([s, sink[h].expand(T, 1)], 1)
                y = _softmax_attention(q, kv[0], kv[1], scores).reshape(T, H * D) * torch.sigmoid(h @ d(m + "g").T)
                y = y @ d(m + "o").T
            x = x + _rms(y, 1.0 + d(p + "norm1"))
            f = p + "mlp."
            if n % 2:
                s = torch.softmax(x @ d(f + "router").T, -1)
                at = torch.topk(s + d(f + "correction"), c["top"], -1).indices
                wt = torch.zeros_like(s).scatter(1, at, s.gather(1, at))
                y = x * wt[:, c["experts"]:].sum(1, keepdim=True)
                for e in range(c["experts"]):
                    r = wt[:, e].nonzero()[:, 0]
                    if len(r):
                        y[r] += wt[r, e, None] * (torch.relu(x[r] @ d(f + "e%d.up" % e).T).square() @ d(f + "e%d.down" % e).T)
            else:
                z = x @ d(f + "up").T
                a = d(f + "act")
                y = (a[0] * _rms(z) + a[1] * _rms(z * z) + a[2] * _rms(z * z * z) + a[3]) @ d(f + "down").T
            x = x + _rms(y, 1.0 + d(p + "norm2"))
        return _rms(x[wanted], 1.0 + d("final.norm")) @ d("head").T


def exact(case, seed):
    c = case
    if c["arch"] == "hybrid":
        return None
    plain, rng = _Plain(c), np.random.default_rng(seed)
    if c["kind"] == "batch":
        if c["batch"] * c["context"] > 50000:
            return None
        ids = rng.integers(0, VOCAB, (c["context"] + 1, c["batch"])).astype(np.int32)
        return {"logits": torch.cat([plain(ids[:, b], [c["context"]]) for b in range(c["batch"])])}
    total = c["tokens"] + c.get("context", 0)
    ids = rng.integers(0, VOCAB, total).astype(np.int32)
    if c["kind"] == "steps":
        return {"logits": plain(ids, [total - 1])[0]}
    return {"logits": plain(ids, list(range(total - c["wanted"], total)))}
