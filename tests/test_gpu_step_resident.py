"""The decode step as one resident kernel, against a plain float64 statement and against the same step as a sequence of launches."""
import threading

import numpy as np
import pytest

from nfai_b200 import LlamaModelFactory, NfaiError, _lib, create_synthetic_model, synth

from .test_gpu_prompt_exact import PlainLlama, off

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def factory():
    f = LlamaModelFactory(0)
    yield f
    f.Dispose()


HALF_MAX = 65504.0
SHAPES = {
    # x of 4 pieces, of 16 in four chunks; shares of 13 and 14 rows (boxes of 8, 4 and 2); an odd vocabulary
    "heads of 64": dict(V=2053),
    # 6 pieces; 2 816 columns: five pieces and a half; three query heads a KV head
    "heads of 128": dict(H=3072, qH=24, kvH=8, d=128, F=2816, V=1111),
    # 8 pieces, the most that are kept; one matrix of fewer columns than rows are dealt to
    "eight pieces": dict(H=4096, qH=16, kvH=8, d=64, F=1536, V=777, tied=False),
    # 3 pieces, one block of columns over 16 pieces; heads of 32 and eight of them a KV head
    "heads of 32": dict(H=1536, qH=32, kvH=4, d=32, F=8256, V=512),
}


class PlainLlamaInFloat16Cache(PlainLlama):
    """The statement with the step's own keys and values as the cache holds them."""

    def attend(self, q, k, v, position):
        k, v = (torch.cat((t[:position], t[position:].half().double())) for t in (k, v))
        return super().attend(q, k, v, position)


@pytest.mark.parametrize("shape,cache,position,ctx", [
    ("heads of 64", "f16", 0, 64), ("heads of 64", "f16", 4094, 4096), ("heads of 128", "f16", 1030, 2048), ("eight pieces", "f16", 63, 128),
    ("heads of 64", "f32", 0, 64), ("heads of 64", "f16", 127, 256), ("heads of 64", "f32", 128, 256), ("heads of 64", "f16", 256, 1024),
    ("heads of 64", "f16", 257, 4096), ("heads of 64", "f32", 4094, 4096), ("heads of 128", "f32", 1, 64), ("heads of 128", "f16", 128, 1024),
    ("heads of 128", "f32", 1030, 2048), ("heads of 128", "f16", 3070, 4096), ("eight pieces", "f32", 63, 128), ("heads of 32", "f32", 300, 512),
    ("heads of 32", "f16", 511, 1024)])
def test_step(factory, shape, cache, position, ctx):
    """Weights are multiplied exactly and summed in float32, as are scores and values. The angles of the rotation are products rounded
    to float32: off by up to position * 2^-24. A float16 cache turns a difference of delta in its newest row into one of 2^-11 in
    delta * 2^11 of its elements, sqrt(delta * 2^-11) of the row, and the second layer's cache does the same to what the first
    passes on, less than it has (1.9e-4 seen at position 63, where that is 1.5e-4; twice that is allowed). A float32 cache is served by
    the sequence of launches."""
    cfg = synth.get_config("s1", gain_std=0.1, **SHAPES[shape])
    delta = 1e-6 + position * 2.0 ** -24
    bound = 1e-5 + position * 2.0 ** -24 if cache == "f32" else 2 * ((delta * 2.0 ** -11) ** 0.5 * 2.0 ** -11) ** 0.5
    rng = np.random.default_rng(position)
    rows = [tuple(rng.standard_normal((position, cfg.kvDim)).astype(np.float16).astype(np.float32) for _ in "kv") for _ in range(cfg.L)]
    m = create_synthetic_model(cfg, ctx, factory=factory, kv_dtype=cache)
    assert (m.step_kernels() == 1) == (cache == "f16")
    if position:
        for l in range(cfg.L):
            m.write_kv_range(l, 0, *rows[l])
        m.set_position(position)
    assert (m.step_kernels() == 1) == (cache == "f16" and (cfg.d < 128 or position < 3072))
    plain, worst = (PlainLlama if cache == "f32" else PlainLlamaInFloat16Cache)(cfg), {}
    for i, token in enumerate(synth.prompt_ids(cfg, 2, 5)):
        new, streams, want = plain.prompt([token], rows)
        got, best = m.decode(int(token))
        worst[f"logits {i}"] = off(got, want)
        assert best == int(np.argmax(got))
        for l in range(cfg.L):
            k, v = m.read_kv(l, position + i)
            if cache == "f16":
                new[l] = tuple(t.half().double() for t in new[l])
            worst[f"rows {i} {l}"] = max(off(k, new[l][0][0]), off(v, new[l][1][0]))
            worst[f"stream {i} {l}"] = off(m.read_hidden(l), streams[l])
        rows = [tuple(np.concatenate((old, t.float().cpu().numpy())) for old, t in zip(rows[l], new[l])) for l in range(cfg.L)]
    m.Dispose()
    assert max(worst.values()) < bound, worst


def test_loops_prompts_and_shapes(factory):
    """Greedy loops repeat bit for bit, prompts too short for a pass go through steps without a head, and a model whose launch shapes
    were asked for runs the launches they belong to."""
    cfg = synth.get_config("s1", V=2053)
    m = create_synthetic_model(cfg, 512, factory=factory)
    ids = synth.prompt_ids(cfg, 5, 0)
    runs = []
    for _ in range(2):
        m.reset()
        first, best = m.prefill(ids)
        tokens, _ = m.decode_greedy(best, 40)
        last, _ = m.decode(tokens[-1])
        runs.append((first.view(np.uint32).tolist(), list(tokens), last.view(np.uint32).tolist()))
    assert runs[0] == runs[1]
    m.reset()
    for token in ids:
        stepped, _ = m.decode(int(token))
    assert np.array_equal(first.view(np.uint32), stepped.view(np.uint32))
    m.tune("ffn_gate_up", 0, 2, 4, 2)
    assert m.step_kernels() == m.step_launches()
    m.reset()
    again, best2 = m.prefill(ids)
    # the cache is of float16: rows that lie between two of its numbers go either way
    assert best2 == best and float(np.linalg.norm(again - first) / np.linalg.norm(first)) < 1e-3
    m.Dispose()


def test_extreme_inputs(factory):
    """Streams that no float16 holds, rows next to nothing, and a layer that makes infinities: as the launches have them."""
    cfg = synth.get_config("s1", V=2053)
    logits = []
    for shaped in (False, True):
        m = create_synthetic_model(cfg, 64, factory=factory, kv_dtype="f16")
        if shaped:
            m.tune("ffn_gate_up", 0, 2, 4, 2)
        rng = np.random.default_rng(0)
        k = rng.standard_normal((8, cfg.kvDim)).astype(np.float32)
        v = np.tile(np.where(rng.random(cfg.kvDim) < 0.5, -6e4, 6e4).astype(np.float32), (8, 1))
        for l in range(cfg.L):
            m.write_kv_range(l, 0, k, v if l == 0 else v * 1e-11)
        m.set_position(8)
        assert (m.step_kernels() == 1) != shaped
        large = m.decode(3)[0]
        assert np.abs(m.read_hidden(0)).max() > HALF_MAX
        v[0, 0] = np.inf
        m.write_kv_range(0, 0, k, v)
        m.set_position(8)
        logits.append((large, m.decode(3)[0]))
        m.Dispose()
    # (the newest row of the second layer's cache, one of nine: sqrt(1e-6 * 2^-11) where the streams differ by 1e-6)
    assert np.isfinite(logits[0][0]).all() and float(np.linalg.norm(logits[0][0] - logits[1][0]) / np.linalg.norm(logits[1][0])) < 2.5e-5
    assert not np.isfinite(logits[0][1]).any() and not np.isfinite(logits[1][1]).any()


def test_a_wait_that_runs_out_is_a_status(factory):
    """With a budget of a nanosecond a step's CTAs give up on one another: the kernel returns, the call says so, and nothing of it is
    left for the next step. Launches have nothing to wait for."""
    def budget(ns):
        _lib.check(_lib.load().nfai_ctx_set_wait_ns(factory.ctx.handle, ns), factory.ctx.handle)

    cfg = synth.get_config("s1", V=2053)
    m, launches = (create_synthetic_model(c, 256, factory=factory) for c in (cfg, synth.get_config("c0")))
    assert m.step_kernels() == 1 and launches.step_kernels() > 1
    ids = synth.prompt_ids(cfg, 20, 3)
    m.prefill(ids)
    want = m.decode(7)[0]
    answer, _ = m.decode_greedy(9, 6)
    small = launches.decode(7)[0]
    try:
        budget(1)
        for _ in range(4):
            m.set_position(len(ids))
            with pytest.raises(NfaiError) as e:
                m.decode(7)
            assert e.value.code == _lib.ERR_TIMEOUT
        launches.reset()
        assert np.array_equal(launches.decode(7)[0], small)
    finally:
        budget(1_000_000_000)
    m.set_position(len(ids))
    assert np.array_equal(m.decode(7)[0], want)
    assert list(m.decode_greedy(9, 6)[0]) == list(answer)
    m.Dispose()
    launches.Dispose()


def test_a_look_ahead_runs_the_launches_it_belongs_to(factory, monkeypatch):
    """Asked for by a call or from outside, and only as long as it is."""
    cfg = synth.get_config("s1", V=2053)
    m = create_synthetic_model(cfg, 64, factory=factory)
    first = m.decode(3)[0]
    for look, extra in ((1 << 20, 0), (0, 1 << 20), (0, 0)):
        m.set_prefetch(look, extra)
        assert (m.step_kernels() == 1) == (look + extra == 0) and m.step_launches() > 1
    m.reset()
    assert np.array_equal(m.decode(3)[0], first)
    m.Dispose()
    for name in ("NFAI_PF_MB", "NFAI_PF_EXTRA_MB"):
        monkeypatch.setenv(name, "1")
        m = create_synthetic_model(cfg, 64, factory=factory)
        monkeypatch.delenv(name)
        assert m.step_kernels() == m.step_launches()
        m.set_prefetch(0)
        assert m.step_kernels() == 1
        m.Dispose()


@pytest.mark.parametrize("qH,kvH,d", [(32, 8, 64), (24, 8, 128), (32, 8, 128), (64, 8, 64), (64, 16, 32)])
def test_which_step_runs(factory, qH, kvH, d):
    """On either side of the line, where a CTA's share of a head is 65 536 elements: the one kernel and the launches agree to what a
    float16 row that goes either way makes of float32 sums in another order."""
    cfg = synth.get_config("s1", V=2053, qH=qH, kvH=kvH, d=d)
    splits = min(16, torch.cuda.get_device_properties(0).multi_processor_count // qH)
    line = min(65536 * splits // d, 4096)
    rng = np.random.default_rng(line)
    rows = [[rng.standard_normal((line, cfg.kvDim)).astype(np.float32) for _ in "kv"] for _ in range(cfg.L)]
    got = []
    for shaped in (False, True):
        m = create_synthetic_model(cfg, 4096, factory=factory, kv_dtype="f16")
        if shaped:
            m.tune("ffn_gate_up", 0, 2, 4, 2)
        for position in (line - 1, line):
            if position < 4096:
                for l in range(cfg.L):
                    m.write_kv_range(l, 0, *rows[l])
                m.set_position(position)
                assert (m.step_kernels() == 1) == (not shaped and position < line)
                got.append(m.decode(3)[0])
        m.Dispose()
    n = len(got) // 2
    assert all(off(a, torch.from_numpy(b)) < 1e-4 for a, b in zip(got[:n], got[n:]))
    assert n == 1 or np.array_equal(got[1], got[3])


def test_steps_and_prompts_of_two_threads(factory):
    """Two contexts on one GPU, a thread each: every step of one needs all of the GPU's SMs at once, whatever the other has running
    there, and waits for them; results are those of either alone."""
    cfg = synth.get_config("s1", V=2053)
    other = LlamaModelFactory(0)
    models = [create_synthetic_model(cfg, 512, factory=f) for f in (factory, other)]
    prompts = [synth.prompt_ids(cfg, n, 4) for n in (5, 160)]

    def work(m, ids, rounds):
        out = []
        for _ in range(rounds):
            m.reset()
            _, best = m.prefill(ids)
            answer, _ = m.decode_greedy(best, 60)
            out.append([list(answer)] + [m.decode(int(t))[0].tolist() for t in ids[:5]])
        return out

    want = [work(m, ids, 1)[0] for m, ids in zip(models, prompts)]
    got, failed = [None, None], []

    def run(i):
        try:
            got[i] = work(models[i], prompts[i], 6)
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not failed and all(g == [w] * 6 for g, w in zip(got, want))
    for m in models:
        m.Dispose()
    other.Dispose()
