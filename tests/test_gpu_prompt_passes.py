"""How a long prompt is divided into passes: by the model, the context and the device, not by what else the device holds."""
import numpy as np
import pytest

from nfai_b200 import LlamaModelFactory, create_synthetic_model, synth

from .gpu_util import rel_err

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def factory():
    f = LlamaModelFactory(0)
    yield f
    f.Dispose()


def ingest(factory, cfg, ctx, ids, leave=None):
    """Logits and some cache rows of a model loaded while the device has `leave` bytes free (None: all it has)."""
    torch.cuda.empty_cache()
    rest = None if leave is None else torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    m = create_synthetic_model(cfg, ctx, factory=factory)
    try:
        out = [m.prefill(ids)[0]]
        for l in range(cfg.L):
            for p in (0, 2047, 2048, len(ids) - 1):
                out += m.read_kv(l, p)
            out.append(m.read_hidden(l))
    finally:
        m.Dispose()
        del rest
        torch.cuda.empty_cache()
    return out


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_passes_do_not_depend_on_free_memory(factory, monkeypatch):
    cfg = synth.get_config("s1")  # (280 MB of weights, 240 of caches and workspaces)
    ids = synth.prompt_ids(cfg, 2400, 4)  # (the last 352 by themselves would have their products split along K)
    want = ingest(factory, cfg, 4096, ids)
    assert same(ingest(factory, cfg, 4096, ids, leave=1200 << 20), want)
    monkeypatch.setenv("NFAI_PREFILL_CHUNK", "2048")
    assert not same(ingest(factory, cfg, 4096, ids), want)  # (it would have shown)


def test_short_passes_where_the_long_workspace_does_not_fit(factory, monkeypatch):
    """After the weights about 340 MB are left: the workspace of 9 472 tokens (466 MB) does not fit, that of 2 048 (101 MB) does."""
    cfg = synth.get_config("s1")
    ids = synth.prompt_ids(cfg, 2500, 5)
    got = ingest(factory, cfg, 9472, ids, leave=620 << 20)
    monkeypatch.setenv("NFAI_PREFILL_CHUNK", "2048")
    assert same(got, ingest(factory, cfg, 9472, ids))


def test_prompt_longer_than_a_pass(factory, monkeypatch):
    """9 472 tokens and 128 more, against passes of 2 048 (each compared with the token-by-token path elsewhere)."""
    cfg = synth.get_config("s3", gain_std=0.1)
    ids = synth.prompt_ids(cfg, 9600, 6)
    out = {}
    for chunk in ("", "2048"):
        monkeypatch.setenv("NFAI_PREFILL_CHUNK", chunk)
        m = create_synthetic_model(cfg, 9600, factory=factory)
        out[chunk] = [m.prefill(ids)[0]] + [m.read_hidden(l) for l in range(cfg.L)]
        for l in range(cfg.L):
            for p in (0, 2047, 2048, 9471, 9472, 9599):
                out[chunk] += m.read_kv(l, p)
        m.Dispose()
    for a, b in zip(out[""], out["2048"]):
        assert np.isfinite(a).all()
        assert rel_err(a, b) < 2e-3  # (float32 sums in another order, rounded to float16 between the kernels: a few 2^-11)
