"""Prompts wide and long enough for the product of two SMs under every epilogue, against plain float64 statements: cache rows,
residual streams and logits."""
import numpy as np
import pytest

from nfai_b200 import LlamaModelFactory, PlannedModel, create_synthetic_model, synth

from . import plain_tometar, plain_tutizen, tometar_util, tutizen_util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def factory():
    f = LlamaModelFactory(0)
    yield f
    f.Dispose()


class PlainLlama:
    """One prompt behind given cache rows, in 64 bits."""

    def __init__(self, cfg, seed=0):
        self.c = cfg
        self.W = {n: torch.from_numpy(synth.gen_tensor(cfg, n, ne, dt, seed)).cuda().double() for n, ne, dt in synth.tensor_specs(cfg)}

    def norm(self, x, name):
        return x / (x.pow(2).mean(-1, keepdim=True) + self.c.eps).sqrt() * self.W[name]

    def rotate(self, x, position):
        half = self.c.ropeDim // 2
        p = torch.arange(position, position + len(x), device="cuda", dtype=torch.float64)
        a = p[:, None] * self.c.rope_theta ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
        cos, sin = a.cos()[:, None], a.sin()[:, None]
        x = x.reshape(len(x), -1, half, 2)
        return torch.stack((cos * x[..., 0] - sin * x[..., 1], sin * x[..., 0] + cos * x[..., 1]), -1).flatten(2)

    def attend(self, q, k, v, position):  # [T][qH][d], [n][kvH][d]
        group = self.c.qH // self.c.kvH
        out = torch.empty_like(q)
        sees = torch.arange(len(k), device="cuda")[None] <= torch.arange(position, position + len(q), device="cuda")[:, None]
        for h in range(self.c.qH):
            s = q[:, h] @ k[:, h // group].T / self.c.d ** 0.5
            out[:, h] = s.masked_fill(~sees, float("-inf")).softmax(-1) @ v[:, h // group]
        return out.flatten(1)

    def prompt(self, ids, rows):
        """rows: per layer the (k, v) rows so far. Returns the layers' new rows, the last token's stream after each layer, its logits."""
        c, position = self.c, len(rows[0][0])
        x = self.W["token_embd.weight"][torch.from_numpy(np.asarray(ids, np.int64)).cuda()]
        new, streams = [], []
        for i in range(c.L):
            b = f"blk.{i}."
            h = self.norm(x, b + "attn_norm.weight")
            q, k, v = (h @ self.W[b + f"attn_{n}.weight"].T for n in "qkv")
            q, k = self.rotate(q, position), self.rotate(k, position).flatten(1)
            new.append((k, v))
            k, v = (torch.cat((torch.from_numpy(old).cuda().double(), t)).reshape(-1, c.kvH, c.d) for old, t in zip(rows[i], (k, v)))
            x = x + self.attend(q, k, v, position) @ self.W[b + "attn_output.weight"].T
            h = self.norm(x, b + "ffn_norm.weight")
            g, u = (h @ self.W[b + f"ffn_{n}.weight"].T for n in ("gate", "up"))
            x = x + (torch.nn.functional.silu(g) * u) @ self.W[b + "ffn_down.weight"].T
            streams.append(x[-1])
        return new, streams, self.norm(x[-1], "output_norm.weight") @ self.W["token_embd.weight" if c.tied else "output.weight"].T


def off(got, want):
    want = want.cpu().numpy()
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


WIDE = dict(qH=24, kvH=8, d=128, H=1024, F=8192, V=2048)  # heads of 128, products of 5 120 and 16 384 columns


@pytest.mark.parametrize("key,over,position,tokens,cache", [
    ("s1", {}, 77, 1601, "f16"),   # every product of a layer in pairs; 13 rows of tiles, the last of 65 rows
    ("s1", {}, 77, 1601, "f32"),   # the same into float32 rows, attention of the warp-level kernel
    ("s1", {}, 1000, 40, "f16"),   # products split along K
    ("s2", WIDE, 300, 700, "f16"),
    ("s2", WIDE, 0, 449, "f16"),
    ("s3", {"qH": 5, "kvH": 1, "H": 320}, 383, 129, "f16")])
def test_llama_prompt(factory, key, over, position, tokens, cache):
    """Float16 activations between the kernels: 2^-11 at each of a layer's seven roundings, in 2-norm 9e-4 measured after two layers."""
    cfg = synth.get_config(key, gain_std=0.1, **over)
    rng = np.random.default_rng(position + tokens)
    rows = [tuple(rng.standard_normal((position, cfg.kvDim)).astype(np.float16).astype(np.float32) for _ in "kv") for _ in range(cfg.L)]
    ids = synth.prompt_ids(cfg, tokens, 11)
    new, streams, logits = PlainLlama(cfg).prompt(ids, rows)
    m = create_synthetic_model(cfg, position + tokens, factory=factory, kv_dtype=cache)
    if position:
        for l in range(cfg.L):
            m.write_kv_range(l, 0, *rows[l])
        m.set_position(position)
    got = m.prefill(ids)[0]
    worst = {"logits": off(got, logits)}
    for l in range(cfg.L):
        worst[f"stream {l}"] = off(m.read_hidden(l), streams[l])
        for p in sorted({0, 1, 31, 32, 63, 127, 128, tokens // 2, tokens - 2, tokens - 1} & set(range(tokens))):
            k, v = m.read_kv(l, position + p)
            worst[f"k {l}"] = max(worst.get(f"k {l}", 0), off(k, new[l][0][p]))
            worst[f"v {l}"] = max(worst.get(f"v {l}", 0), off(v, new[l][1][p]))
    m.Dispose()
    assert max(worst.values()) < 4e-3, worst


PLANS = {
    # 12 576 columns of queries, keys, values and gates with a bias; 16 384 clamped gate/up columns; 16 400 with router logits behind
    "tutizen": (tutizen_util, plain_tutizen, tutizen_util.config([
        tutizen_util.layer(tutizen_util.attn(96, 1, 128, 64), tutizen_util.dense(8192)),
        tutizen_util.layer(tutizen_util.attn(4, 2, 32, 48), tutizen_util.moe(12, 3, 40, 8200, 3, 2))], 256, 200)),
    # 13 392 columns of queries, latents and gates, keys and values of 12 288 from latents of 64, 16 384 gate/up columns with a bias,
    # 12 448 into a recurrent layer
    "tometar": (tometar_util, plain_tometar, tometar_util.config([
        tometar_util.layer(tometar_util.latent(64, 96, 16, 96, 64, 150), 8192),
        tometar_util.layer(tometar_util.ssm(96, 64, 16, 2, 4, 4))], 128, 200, 2)),
}


@pytest.mark.parametrize("name", PLANS)
def test_wide_plan_prompt(cuda_ctx, name):
    """150 tokens: two rows of tiles, so that the products above go to pairs. Bfloat16 activations: 2^-8 at each rounding, 5e-3 measured."""
    U, plain, cfg = PLANS[name]
    W = U.weights(cfg)
    toks = tutizen_util.tokens(cfg, W, 150, 100) if name == "tutizen" else np.random.default_rng(100).integers(0, cfg["vocab"], 150).tolist()
    taps = []
    want = plain.forward(cfg, {k: v.astype(np.float64) for k, v in W.items()}, toks, taps=taps)
    m = PlannedModel.from_tensors(cuda_ctx, cfg, U.tensors(W), 160, "bf16")
    places = list(range(0, 150, 7)) + [149]
    worst = [U.error(m.forward(toks, places), want[places])] + [U.error(m.read_hidden(l), np.array(taps)[-1, l]) for l in range(m.L)]
    m.Dispose()
    assert max(worst) < 2e-2, worst
