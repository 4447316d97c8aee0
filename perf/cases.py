"""The work that programs have this framework do, as cases that can be timed and checked one by one.

One model on one GPU, batch 1, through the public step functions (`prefill`, `decode`, `decode_greedy`): a prompt comes in,
tokens go out. The models are the ones of nfai_b200/synth.py and of the benchmark's two other designs, with random weights.
A case is a model, a cache size, a position the conversation has reached, and one of

  greedy   `tokens` steps of the device-side loop, then the step whose logits the program looks at
  steps    `tokens` per-token calls with tokens that the host picks, the logits of the last one read back
  prompt   `tokens` prompt tokens at once, the last one's logits read back

A program loads a model once and then serves inputs, so a process keeps the models it has loaded (Loaded below); what a seed
decides is the tokens. The rows of the conversation so far are the same for all passes of a case.
"""
from __future__ import annotations

import math
import zlib
from collections import OrderedDict

import numpy as np
import torch

import nfai_b200
from nfai_b200 import _lib, synth
from nfai_b200.gguf_io import ComputeCollection

# ---- models --------------------------------------------------------------------------------------------------------
LLAMA = {"llama-tiny-f32": "c0", "llama-1b": "c1", "llama-3b": "c2", "llama-8b": "c3"}

_TOMETAR_LATENT = dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, mask={"size": 1024},
                       rot={"base": 500000.0, "dims": 64}, scale=192 ** -0.5)
_TOMETAR_SSM = dict(heads=64, vdim=64, state=128, groups=8, conv=4, norm_groups=8)
_TUTIZEN_ATTN = dict(heads=32, kv_heads=8, dim=64, vdim=64, scale=64 ** -0.5)
_TUTIZEN_MOE = {"kind": "moe", "expert": {"ff": 1536, "limit": 7.0}, "shared": {"ff": 2048, "limit": 7.0},
                "router": {"experts": 32, "top": 4, "scale": 2.5, "groups": {"count": 4, "keep": 2}}}
PLANS = {
    # latent attention and state space layers in turn, all with a feed-forward
    "tometar-1b": {"architecture": "Tometar", "norm": {"eps": 1e-5}, "streams": 4, "vocab": 128256, "width": 2048, "layers": [
        {"type": "latent_attention", "mixer": _TOMETAR_LATENT, "mlp": {"kind": "dense", "ff": 8192}} if i % 2 == 0 else
        {"type": "mamba2", "mixer": _TOMETAR_SSM, "mlp": {"kind": "dense", "ff": 8192}} for i in range(16)]},
    # dense layers with keys of their own and routed layers that borrow them, in turn
    "tutizen-1b": {"architecture": "Tutizen", "norm": {"eps": 1e-5}, "residual_mult": 0.5, "vocab": 128256, "width": 2048, "layers": [
        {"type": "attention", "mixer": _TUTIZEN_ATTN, "mlp": {"kind": "dense", "ff": 8192, "limit": 7.0}} if i % 2 == 0 else
        {"type": "attention", "mixer": dict(_TUTIZEN_ATTN, kv_from=i - 1), "mlp": _TUTIZEN_MOE} for i in range(16)]},
}


def listed():
    return [
        # the smallest model there is, one token per call: host calls and launches are all there is
        {"name": "tiny-f32-steps", "model": "llama-tiny-f32", "kind": "steps", "ctx": 256, "position": 64, "tokens": 16},
        # an answer early in a chat: the plain case of local inference
        {"name": "1b-chat", "model": "llama-1b", "kind": "greedy", "ctx": 1024, "position": 128, "tokens": 15},
        # the same with the largest of the models, further on
        {"name": "8b-chat", "model": "llama-8b", "kind": "greedy", "ctx": 2048, "position": 1030, "tokens": 7},
        # an answer about a long document: attention over 32 768 positions
        {"name": "1b-long-steps", "model": "llama-1b", "kind": "steps", "ctx": 32832, "position": 32768, "tokens": 8},
        # the user's next message in a chat
        {"name": "1b-turn-37", "model": "llama-1b", "kind": "prompt", "ctx": 1024, "position": 603, "tokens": 37},
        # a question with a little context
        {"name": "1b-prompt-128", "model": "llama-1b", "kind": "prompt", "ctx": 1024, "position": 0, "tokens": 128},
        # a page or two of text, not a round number of tokens
        {"name": "3b-prompt-2011", "model": "llama-3b", "kind": "prompt", "ctx": 4096, "position": 0, "tokens": 2011},
        # a long document
        {"name": "1b-prompt-30011", "model": "llama-1b", "kind": "prompt", "ctx": 32832, "position": 0, "tokens": 30011},
        # the other designs: generation and ingestion
        {"name": "tometar-steps", "model": "tometar-1b", "kind": "steps", "ctx": 2112, "position": 509, "tokens": 8},
        {"name": "tometar-prompt-2011", "model": "tometar-1b", "kind": "prompt", "ctx": 2112, "position": 0, "tokens": 2011},
        {"name": "tutizen-steps", "model": "tutizen-1b", "kind": "steps", "ctx": 2112, "position": 509, "tokens": 8},
        {"name": "tutizen-prompt-2011", "model": "tutizen-1b", "kind": "prompt", "ctx": 2112, "position": 0, "tokens": 2011},
    ]


def draw(rng):
    """Models by how much they are used, lengths even over their logarithm."""
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["llama-tiny-f32", "llama-1b", "llama-1b", "llama-1b", "llama-3b", "llama-8b", "tometar-1b", "tutizen-1b"])
    most = {"llama-tiny-f32": 250, "llama-1b": 30000, "llama-3b": 4000, "llama-8b": 2000}.get(model, 2048)
    if rng.random() < 0.5:  # ingestion, half of it in a conversation that has begun
        tokens = between(8, most)
        room = min(most - tokens, 4000)
        position = between(1, room) if room > 1 and model in LLAMA and rng.random() < 0.5 else 0
        kind = "prompt"
    else:
        tokens = rng.randint(2, 20)
        position = between(8, most - tokens - 1)
        kind = rng.choice(["greedy", "steps"]) if model in LLAMA else "steps"
    need = position + tokens + 1
    ctx = next(c for c in ((256,) if model == "llama-tiny-f32" else (2112,) if model in PLANS else (1024, 2048, 4096, 32832)) if c >= need)
    return {"model": model, "kind": kind, "ctx": ctx, "position": position, "tokens": tokens}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _normal(key, shape):
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(key.encode()))
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)


def llama_weight(model, name, shape):
    """[out][in] as stored; gains are one."""
    if name.endswith("_norm.weight"):
        return torch.ones(shape, device="cuda", dtype=torch.float32)
    w = _normal(model + name, shape) * 0.02
    return w.half() if synth.get_config(LLAMA[model]).dtype == "f16" else w


def plan_weight(model, name, shape):
    """bfloat16. Tutizen's routers read a quarter of the coordinates that no sublayer writes, so that a token's experts follow from
    the token and its position, as firmly in 16 as in 64 bits."""
    cfg, last = PLANS[model], name.split(".")[-1]
    n = _normal(model + name, shape)
    if last.startswith("norm"):
        w = 1.0 + 0.1 * n
    elif ".hc" in name:
        w = torch.eye(shape[0], device="cuda") * 0.9 + 0.1 * n if last == "mix" else 1.0 / shape[0] + 0.05 * n if last == "in" else 0.8 + 0.2 * n
    elif last == "A_log":
        w = torch.linspace(0.0, 2.7, shape[0], device="cuda")
    elif last == "dt_bias":
        w = -4.0 + 0.3 * n
    elif last == "D":
        w = 1.0 + 0.3 * n
    elif last == "conv":
        w = 0.5 * n
    elif last in ("b", "correction"):
        w = 0.02 * n
    elif name == "embed":
        w = n
    else:
        w = n / math.sqrt(shape[-1])
    if cfg["architecture"] == "Tometar" and last in ("o", "down"):  # (a residual is mostly what the layers before have left)
        w = w / math.sqrt(2 * len(cfg["layers"]))
    if cfg["architecture"] == "Tutizen":
        own = cfg["width"] // 4
        if last == "router":
            w = 2.0 * w
            w[:, own:] = 0
        elif last in ("o", "down") or name.endswith("o.b"):
            w[:own] = 0
    return w.bfloat16()


def context_rows(model, layer, which, n, width):
    """What the cache holds of the conversation so far: rows as large as the model's own, exact in float16."""
    return (_normal(f"{model} cache {layer} {which}", (n, width)) * 0.9).half()


def token_ids(model, seed, n):
    return np.random.default_rng(seed).integers(0, vocab(model), n)


def vocab(model):
    return synth.get_config(LLAMA[model]).V if model in LLAMA else PLANS[model]["vocab"]


def history(case):
    """Prompt of a layer-plan model's conversation so far (its cache is only ever written by the model itself)."""
    return token_ids(case["model"], 1, case["position"])


# ---- the framework's side --------------------------------------------------------------------------------------------
class _Tensor(ComputeCollection):
    """A weight that is made when the model asks for it."""

    def __init__(self, model, name, ne, dtype):
        super().__init__(name, ne, 2 if dtype == "f16" else 4)
        self._model = model

    def get_data_raw(self, widen_half=False):
        self._array = llama_weight(self._model, self.Name, tuple(reversed(self.Shape))).cpu().numpy()
        try:
            yield from super().get_data_raw(widen_half=widen_half)
        finally:
            self._array = None


class Loaded:
    """A model in GPU memory, and what its cache holds at the moment."""

    context = None
    models = OrderedDict()  # (model, cache size) -> Loaded, least recently used first

    def __init__(self, name, ctx_size):
        if Loaded.context is None:
            Loaded.context = nfai_b200.CudaContext(0)
        if name in LLAMA:
            cfg = synth.get_config(LLAMA[name])
            tensors = [_Tensor(name, n, ne, dt) for n, ne, dt in synth.tensor_specs(cfg)]
            self.model = nfai_b200.LlamaModel(Loaded.context, synth.metadata(cfg), tensors, ctx_size)
        else:
            tensors = ((n, plan_weight(name, n, s).view(torch.uint16).cpu().numpy(), _lib.BF16)
                       for n, s in nfai_b200.config_tensors(PLANS[name]).items())
            self.model = nfai_b200.PlannedModel.from_tensors(Loaded.context, PLANS[name], tensors, ctx_size, "bf16")
        self.holds = None
        self.snapshot = None

    @classmethod
    def get(cls, name, ctx_size):
        key = (name, ctx_size)
        if key not in cls.models:
            while len(cls.models) >= 7:  # (about 50 GB at most)
                cls.models.popitem(last=False)
            cls.models[key] = cls(name, ctx_size)
        cls.models.move_to_end(key)
        return cls.models[key]

    def hold(self, case):
        """Bring the conversation of a case into the cache."""
        m, pos, want = self.model, case["position"], (case["kind"], case["position"])
        if self.holds == want:
            return
        if self.snapshot is not None:
            self.snapshot.close()
            self.snapshot = None
        if case["model"] in LLAMA:
            if pos:
                width = m.hp.kvH * m.hp.d
                for layer in range(m.L):
                    k, v = (context_rows(case["model"], layer, w, pos, width).float().cpu().numpy() for w in "kv")
                    m.write_kv_range(layer, 0, k, v)
        else:
            m.reset()
            if pos:
                m.prefill(history(case), want_logits=False)
                self.snapshot = m.snapshot()
        self.holds = want


def prepare(case, seed):
    loaded = Loaded.get(case["model"], case["ctx"])
    loaded.hold(case)
    return {"model": loaded.model, "kind": case["kind"], "position": case["position"], "snapshot": loaded.snapshot,
            "tokens": token_ids(case["model"], seed, case["tokens"]), "loaded": loaded}


def run(state):
    m, tokens = state["model"], state["tokens"]
    if state["snapshot"] is not None:
        state["snapshot"].restore()
    else:
        m.set_position(state["position"])
    if state["kind"] == "prompt":
        return m.prefill(tokens)[0]
    if state["kind"] == "greedy":
        answer, _ = m.decode_greedy(tokens[0], len(tokens))
        logits, _ = m.decode(answer[-1])
        return {"tokens": answer, "logits": logits}
    for t in tokens[:-1]:
        m.decode(t, want_logits=False)
    return m.decode(tokens[-1])[0]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _layer_sizes(model):
    """Per layer: matrix elements that one token uses, matrix elements a long prompt uses, cache bytes per position, attention
    multiply-adds per (query, position), and how far back a query looks (None: to the start)."""
    if model in LLAMA:
        c = synth.get_config(LLAMA[model])
        p = c.H * (2 * c.qDim + 2 * c.kvDim + 3 * c.F)
        return [(p, p, 2 * c.kvDim * (2 if c.dtype == "f16" else 4), 2 * c.qDim, None)] * c.L
    cfg, out = PLANS[model], []
    for layer in cfg["layers"]:
        m, f, H = layer["mixer"], layer["mlp"], cfg["width"]
        ff = 3 * H * f["ff"] if f["kind"] == "dense" else 0
        if layer["type"] == "latent_attention":
            p = H * (m["heads"] * (m["dim"] + m["rot_dim"] + 2 * m["vdim"]) + m["kv_rank"] + m["rot_dim"]) + m["heads"] * (m["dim"] + m["vdim"]) * m["kv_rank"]
            out.append((p + ff, p + ff, 2 * (m["kv_rank"] + m["rot_dim"]), m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["mask"]["size"]))
        elif layer["type"] == "mamba2":
            p = H * (3 * m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"] + m["heads"])
            out.append((p + ff, p + ff, 0, 2 * m["heads"] * m["vdim"] * m["state"], 1))
        else:
            p = H * m["heads"] * (m["dim"] + m["vdim"] + 1)
            rows = 2 * m["kv_heads"] * (m["dim"] + m["vdim"])
            if m.get("kv_from") is None:
                p += H * m["kv_heads"] * (m["dim"] + m["vdim"])
            used = whole = ff
            if f["kind"] == "moe":
                shared = 3 * H * f["shared"]["ff"] + H * (f["router"]["experts"] + 1)
                used = 3 * H * f["router"]["top"] * f["expert"]["ff"] + shared
                whole = 3 * H * f["router"]["experts"] * f["expert"]["ff"] + shared
            out.append((p + used, p + whole, rows, m["heads"] * (m["dim"] + m["vdim"]), None))
    return out


def work(case):
    model, n, pos = case["model"], case["tokens"], case["position"]
    H = synth.get_config(LLAMA[model]).H if model in LLAMA else PLANS[model]["width"]
    size = 4 if model == "llama-tiny-f32" else 2
    steps = case["kind"] != "prompt"
    if case["kind"] == "greedy":
        n += 1
    head = vocab(model) * H
    nbytes = (n if steps else 1) * head * size + n * H * size + vocab(model) * 4
    flops = 2.0 * head * (n if steps else 1)
    for used, whole, row, pair, back in _layer_sizes(model):
        seen = sum(min(pos + i + 1, back or pos + n) for i in range(n))  # (query, position) pairs
        first = min(pos, back or pos)
        nbytes += used * size * n + row * (seen + n) if steps else min(whole, used * n) * size + row * (first + n)
        flops += 2.0 * used * n + 2.0 * pair * seen
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """About four times what the paths differ by from exact() (relative, of the logits)."""
    if case["model"] == "llama-tiny-f32":
        return {"rel": 2e-6}
    if case["model"] in PLANS:  # bfloat16 operands and caches: up to 1.4e-2 and 5e-3
        return {"rel": 3e-2 if case["model"] == "tometar-1b" else 2e-2}
    return {"rel": 1e-2 if case["kind"] == "prompt" else 3e-3}


# ---- 64-bit statement ----------------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, first, window=None, slopes=None):
    """q [T][heads][d] at positions first.., k and v [positions][groups][..] from position 0; causal. -> [T][heads][dv]"""
    T, heads = q.shape[:2]
    share = heads // k.shape[1]
    out = torch.empty(T, heads, v.shape[2], device="cuda", dtype=torch.float64)
    for a in range(0, T, 2048):
        b = min(T, a + 2048)
        lo, hi = max(0, first + a + 1 - (window or 1 << 40)), first + b
        back = torch.arange(first + a, first + b, device="cuda")[:, None] - torch.arange(lo, hi, device="cuda")[None]
        gone = (back < 0) | (back >= (window or 1 << 40))
        for h in range(heads):
            s = q[a:b, h] @ k[lo:hi, h // share].T * scale
            if slopes is not None:
                s -= slopes[h] * back
            out[a:b, h] = torch.softmax(s.masked_fill_(gone, -math.inf), -1) @ v[lo:hi, h // share]
    return out


class _ExactLlama:
    def __init__(self, case):
        self.name, self.c, self.pos = case["model"], synth.get_config(LLAMA[case["model"]]), case["position"]
        c, n = self.c, case["position"]
        self.kv = [[context_rows(self.name, i, w, n, c.kvDim).double() if n else torch.empty(0, c.kvDim, device="cuda", dtype=torch.float64)
                    for w in "kv"] for i in range(c.L)]
        self.weights = {n: llama_weight(self.name, n, tuple(reversed(ne))) for n, ne, _ in synth.tensor_specs(c)}

    def w(self, name):
        return self.weights[name + ".weight"].double()

    def rope(self, x):
        half = self.c.d // 2
        p = torch.arange(self.pos, self.pos + x.shape[0], device="cuda", dtype=torch.float64)
        a = p[:, None] * self.c.rope_theta ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
        cos, sin = a.cos()[:, None], a.sin()[:, None]
        x = x.view(x.shape[0], -1, half, 2)
        return torch.stack((cos * x[..., 0] - sin * x[..., 1], sin * x[..., 0] + cos * x[..., 1]), -1).flatten(2)

    def feed(self, tokens):
        """Logits of the last one."""
        c, T = self.c, len(tokens)
        x = self.weights["token_embd.weight"][torch.as_tensor(np.asarray(tokens, np.int64), device="cuda")].double()
        for i in range(c.L):
            b = f"blk.{i}."
            h = _rms(x, c.eps) * self.w(b + "attn_norm")
            q, k = self.rope((h @ self.w(b + "attn_q").T)), self.rope((h @ self.w(b + "attn_k").T))
            self.kv[i] = [torch.cat((old, new)) for old, new in zip(self.kv[i], (k.flatten(1), h @ self.w(b + "attn_v").T))]
            k, v = (t.view(-1, c.kvH, c.d) for t in self.kv[i])
            x = x + _attend(q, k, v, c.d ** -0.5, self.pos).flatten(1) @ self.w(b + "attn_output").T
            h = _rms(x, c.eps) * self.w(b + "ffn_norm")
            x = x + (torch.nn.functional.silu(h @ self.w(b + "ffn_gate").T) * (h @ self.w(b + "ffn_up").T)) @ self.w(b + "ffn_down").T
        self.pos += T
        return (self.w("token_embd" if c.tied else "output") @ (_rms(x[-1], c.eps) * self.w("output_norm")))


def _exact_tometar(cfg, W, tokens):
    eps, S, T = cfg["norm"]["eps"], cfg["streams"], len(tokens)
    H = cfg["width"]
    X = W("embed", (cfg["vocab"], H), rows=tokens)[None].repeat(S, 1, 1)

    def read(p, hc, norm):
        return _rms(torch.einsum("s,sth->th", W(p + hc + ".in", (S,)), X), eps) * W(p + norm, (H,))

    def write(p, hc, y):
        return torch.einsum("st,sxh->txh", W(p + hc + ".mix", (S, S)), X) + W(p + hc + ".out", (S,))[:, None, None] * y

    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        h = read(p, "hc1", "norm1")
        if layer["type"] == "latent_attention":
            n, d, r, dv, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            a = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * m["rot"]["base"] ** (-2.0 * torch.arange(r // 2, device="cuda", dtype=torch.float64) / r)

            def turn(v):
                lo, hi = v[..., :r // 2], v[..., r // 2:]
                cos, sin = (t.view(T, *[1] * (v.dim() - 2), r // 2) for t in (a.cos(), a.sin()))
                return torch.cat((lo * cos - hi * sin, hi * cos + lo * sin), -1)
            q = (h @ W(p + "mix.q", (n * (d + r), H)).T).view(T, n, d + r)
            kv = h @ W(p + "mix.dkv", (R + r, H)).T
            c = _rms(kv[:, :R], eps) * W(p + "mix.dkv.norm", (R,))
            k = torch.cat(((c @ W(p + "mix.uk", (n * d, R)).T).view(T, n, d), turn(kv[:, R:])[:, None].expand(T, n, r)), -1)
            v = (c @ W(p + "mix.uv", (n * dv, R)).T).view(T, n, dv)
            o = _attend(torch.cat((q[..., :d], turn(q[..., d:])), -1), k, v, m["scale"], 0, m["mask"]["size"])
            y = (o.flatten(1) * torch.sigmoid(h @ W(p + "mix.g", (n * dv, H)).T)) @ W(p + "mix.o", (H, n * dv)).T
        else:
            n, V, N, G, taps = m["heads"], m["vdim"], m["state"], m["groups"], m["conv"]
            inner, ch = n * V, n * V + 2 * G * N
            u = h @ W(p + "mix.in", (inner + ch + n, H)).T
            z, xbc, dt = u[:, :inner], u[:, inner:inner + ch], torch.nn.functional.softplus(u[:, inner + ch:] + W(p + "mix.dt_bias", (n,)))
            past = torch.cat((torch.zeros(taps - 1, ch, device="cuda", dtype=torch.float64), xbc))
            conv = W(p + "mix.conv", (ch, taps))
            xbc = torch.nn.functional.silu(W(p + "mix.conv.b", (ch,)) + sum(conv[:, j] * past[j:j + T] for j in range(taps)))
            x, B, C = xbc[:, :inner].view(T, n, V), xbc[:, inner:inner + G * N].view(T, G, N), xbc[:, inner + G * N:].view(T, G, N)
            B, C = (t.repeat_interleave(n // G, 1) for t in (B, C))
            decay, D = torch.exp(-torch.exp(W(p + "mix.A_log", (n,))) * dt), W(p + "mix.D", (n,))
            state = torch.zeros(n, N, V, device="cuda", dtype=torch.float64)
            out = torch.empty(T, n, V, device="cuda", dtype=torch.float64)
            dx = dt[..., None] * x
            for t in range(T):
                state.mul_(decay[t, :, None, None]).baddbmm_(B[t][:, :, None], dx[t][:, None])
                torch.bmm(C[t][:, None], state, out=out[t][:, None])
            y = ((out + D[:, None] * x).flatten(1) * torch.nn.functional.silu(z)).view(T, m["norm_groups"], -1)
            y = (_rms(y, eps).flatten(1) * W(p + "mix.norm", (inner,))) @ W(p + "mix.o", (H, inner)).T
        X = write(p, "hc1", y)
        h = read(p, "hc2", "norm2")
        gate, up = (h @ W(p + "mlp." + g, (ff, H)).T + W(p + "mlp." + g + ".b", (ff,)) for g in ("gate", "up"))
        X = write(p, "hc2", (torch.relu(gate) * up) @ W(p + "mlp.down", (H, ff)).T + W(p + "mlp.down.b", (H,)))
    return W("head", (cfg["vocab"], H)) @ (_rms(X.sum(0)[-1], eps) * W("final.norm", (H,)))


def _exact_tutizen(cfg, W, tokens):
    eps, mult, T, H = cfg["norm"]["eps"], cfg["residual_mult"], len(tokens), cfg["width"]
    i = torch.arange(H, device="cuda")
    a = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * 10000.0 ** (-2.0 * (i // 2) / H).double()
    x = W("embed", (cfg["vocab"], H), rows=tokens) + torch.where(i % 2 == 0, a.sin(), a.cos())
    past = {}

    def forward(h, p, ff, limit):
        g, u = torch.clamp(h @ W(p + "gate", (ff, H)).T, max=limit), torch.clamp(h @ W(p + "up", (ff, H)).T, -limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W(p + "down", (H, ff)).T

    for n, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{n}.", layer["mixer"], layer["mlp"]
        heads, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]

        def proj(what, parts, width):
            y = x @ W(p + "mix." + what, (parts * width, H)).T + W(p + "mix." + what + ".b", (parts * width,))
            return _rms(y.view(T, parts, width), eps)
        if m.get("kv_from") is None:
            past[n] = proj("k", G, d), proj("v", G, dv)
        k, v = past[m.get("kv_from", n)]
        slopes = 2.0 ** (-8.0 * (torch.arange(heads, device="cuda", dtype=torch.float64) + 1) / heads)
        o = _attend(proj("q", heads, d), k, v, m["scale"], 0, None, slopes) * torch.sigmoid(x @ W(p + "mix.g", (heads, H)).T)[..., None]
        y = o.flatten(1) @ W(p + "mix.o", (H, heads * dv)).T + W(p + "mix.o.b", (H,))
        x = x + mult * _rms(y, eps) * W(p + "norm1", ())
        if f["kind"] == "dense":
            y = forward(x, p + "mlp.", f["ff"], f["limit"])
        else:
            r, E = f["router"], f["router"]["experts"]
            s = torch.sigmoid(x @ W(p + "mlp.router", (E, H)).T)
            c = s + W(p + "mlp.correction", (E,))
            groups = c.view(T, r["groups"]["count"], -1)
            keep = groups.topk(min(2, groups.shape[2]), -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
            allowed = torch.zeros(groups.shape[:2], device="cuda", dtype=torch.bool).scatter_(1, keep, True)
            chosen = c.masked_fill(~allowed.repeat_interleave(groups.shape[2], 1), -math.inf).topk(r["top"], -1).indices
            w = s.gather(1, chosen)
            w = w / (w.sum(-1, keepdim=True) + 1e-20) * r["scale"]
            y = torch.sigmoid(x @ W(p + "mlp.shared.sg", (1, H)).T) * forward(x, p + "mlp.shared.", f["shared"]["ff"], f["shared"]["limit"])
            for e in range(E):
                at, place = (chosen == e).nonzero(as_tuple=True)
                if len(at):
                    y[at] += w[at, place, None] * forward(x[at], f"{p}mlp.e{e}.", f["expert"]["ff"], f["expert"]["limit"])
        x = x + mult * _rms(y, eps) * W(p + "norm2", ())
    return W("head", (cfg["vocab"], H)) @ (_rms(x[-1], eps) * W("final.norm", ()))


def exact(case, seed):
    """What run() returns, in 64 bits and without the framework's code."""
    model, tokens = case["model"], token_ids(case["model"], seed, case["tokens"])
    if model in LLAMA:
        m = _ExactLlama(case)
        if case["kind"] != "greedy":
            return m.feed(tokens).cpu().numpy()
        t, answer = int(tokens[0]), []
        for _ in tokens:
            t = int(m.feed([t]).argmax())
            answer.append(t)
        return {"tokens": np.array(answer, np.uint32), "logits": m.feed([t]).cpu().numpy()}
    cfg = PLANS[model]

    def weight(name, shape, rows=None):
        w = plan_weight(model, name, shape)
        return (w if rows is None else w[torch.as_tensor(rows, device="cuda")]).double()
    every = np.concatenate((history(case), tokens)) if case["position"] else tokens
    return (_exact_tometar if cfg["architecture"] == "Tometar" else _exact_tutizen)(cfg, weight, every).cpu().numpy()
