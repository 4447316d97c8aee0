"""Tiles of the prompt kernels at their edges: products over pairs of SMs against float64 products of the same operands, attention in
tensor memory against the warp-level kernel of the same arithmetic."""
import numpy as np
import pytest

from nfai_b200 import create_synthetic_model, LlamaModel, LlamaModelFactory, synth
from nfai_b200.api import synthetic_tensors

from .gpu_util import call, host, ptr, rel_err

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M,N,K", [(2011, 3072, 200),   # tiles of 192 columns, a ragged last row tile and K step
                                   (1537, 4100, 136),   # one row in the last row tile, a column remainder in quads
                                   (2049, 2050, 64),    # columns in pairs only
                                   (1665, 2051, 72),    # an odd row length
                                   (3072, 2048, 64),    # whole tiles, one K step
                                   (9472, 1024, 64)])   # more tiles than two per pair
def test_pair_tiles(cuda_ctx, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = (torch.randn(M, K, generator=g, device="cuda") * 0.5).half()
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).half()
    C = torch.full((M, N), float("nan"), device="cuda")
    call(cuda_ctx, "nfai_op_gemm_f16", ptr(A), ptr(W), M, N, K, ptr(C))
    want = (A.double() @ W.double().T).cpu().numpy()
    got = host(C)
    assert np.isfinite(got).all()
    assert rel_err(got, want) < 1e-5  # float32 sums of at most 200 products: 200 * 2^-24


@pytest.mark.parametrize("M,N,K", [(128, 2048, 2048), (37, 3072, 2048), (1, 2048, 512), (129, 1026, 520),  # rows that do not divide by the cluster
                                   (16, 2051, 1024), (256, 2048, 1032), (512, 2048, 4096), (70, 130, 4096)])  # the last through memory
def test_split_tiles(cuda_ctx, M, N, K):
    """K divided over the CTAs of a cluster, or over more than fit into one: against a float64 product."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = (torch.randn(M, K, generator=g, device="cuda") * 0.5).half()
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).half()
    C = torch.full((M, N), float("nan"), device="cuda")
    call(cuda_ctx, "nfai_op_gemm_f16", ptr(A), ptr(W), M, N, K, ptr(C))
    got = host(C)
    assert np.isfinite(got).all()
    assert rel_err(got, (A.double() @ W.double().T).cpu().numpy()) < 1e-4  # float32 sums of up to 4096 products


@pytest.mark.parametrize("M,N,K", [(1000, 2012, 136), (1000, 2010, 72),                  # tiles of 128 columns
                                   (640, 2532, 136), (640, 2550, 200),                   # of 64
                                   (100, 516, 64), (77, 518, 64), (33, 77, 64),          # of 32
                                   (45, 132, 1024), (70, 130, 1024), (128, 1028, 1024),  # split, through memory and in clusters
                                   (1537, 4100, 136), (1537, 4098, 136)])                # pairs
def test_columns_that_end_inside_a_block(cuda_ctx, M, N, K):
    """The last block of 32 columns is live in some of a warp's lanes only (in quads and in pairs), in every kernel, mostly with dead
    blocks behind it; nothing is written beyond the product."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = (torch.randn(M, K, generator=g, device="cuda") * 0.5).half()
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).half()
    C = torch.full((M * N + 256,), float("nan"), device="cuda")
    call(cuda_ctx, "nfai_op_gemm_f16", ptr(A), ptr(W), M, N, K, ptr(C))
    got = host(C)
    assert np.isnan(got[M * N:]).all() and np.isfinite(got[:M * N]).all()
    assert rel_err(got[:M * N].reshape(M, N), (A.double() @ W.double().T).cpu().numpy()) < K * 2.0 ** -24


@pytest.fixture(scope="module")
def factory():
    f = LlamaModelFactory(0)
    yield f
    f.Dispose()


@pytest.mark.parametrize("position,tokens", [(0, 257),     # a third tile of one position (the warp-level kernel's at these widths)
                                             (248, 9),     # the fewest tokens, rows of one CTA only in part
                                             (0, 321), (312, 9),  # the same on the tcgen05 kernel
                                             (255, 130),
                                             (383, 33),    # the last position of a tile is the first token's own
                                             (1000, 517)])
@pytest.mark.parametrize("heads,kv_heads,d", [(8, 2, 64), (6, 2, 128), (3, 3, 64), (5, 1, 128)])
def test_attention_tiles(factory, monkeypatch, heads, kv_heads, d, position, tokens):
    """Rows behind the last token are NaN; some keys score far above all before them, so that sums are rescaled on the way."""
    cfg = synth.get_config("s3", qH=heads, kvH=kv_heads, d=d, H=heads * d, gain_std=0.1)
    m = create_synthetic_model(cfg, 1664, factory=factory, kv_dtype="f16")
    rng = np.random.default_rng(position + tokens + heads)
    for layer in range(cfg.L):
        k, v = (rng.standard_normal((1664, cfg.kvDim), dtype=np.float32) for _ in "kv")
        k[100:120] *= 8
        k[200:210] *= 30
        k[position:] = v[position:] = np.nan
        m.write_kv_range(layer, 0, k, v)
    ids = synth.prompt_ids(cfg, tokens, 7)
    out = {}
    for kind in ("1", "2"):
        monkeypatch.setenv("NFAI_PREFILL_ATTN", kind)
        m.set_position(position)
        out[kind] = m.prefill(ids)[0], m.read_hidden(0), m.read_hidden(1)
    m.Dispose()
    for a, b in zip(out["1"], out["2"]):
        assert np.isfinite(a).all()
        assert rel_err(a, b) < 2e-3  # (float32 sums in another order, rounded to float16 between the kernels: a few 2^-11)


@pytest.mark.parametrize("heads,kv_heads,d,tokens,longest", [(8, 2, 64, 40, 320), (32, 8, 64, 191, 320), (32, 8, 64, 192, 256),
                                                             (8, 8, 128, 300, 320), (24, 8, 128, 170, 320), (24, 8, 128, 171, 448)])
def test_which_attention_runs(factory, monkeypatch, heads, kv_heads, d, tokens, longest):
    """On either side of the line to the warp-level kernel: the same bits as that kernel's up to it, others (and close) beyond."""
    cfg = synth.get_config("s3", qH=heads, kvH=kv_heads, d=d, gain_std=0.1)
    m = create_synthetic_model(cfg, 512, factory=factory, kv_dtype="f16")
    rng = np.random.default_rng(heads + tokens)
    ids = synth.prompt_ids(cfg, tokens, 9)
    for positions in (longest, longest + 1):
        for layer in range(cfg.L):
            m.write_kv_range(layer, 0, *(rng.standard_normal((512, cfg.kvDim), dtype=np.float32) for _ in "kv"))
        out = {}
        for kind in ("1", "2"):
            monkeypatch.setenv("NFAI_PREFILL_ATTN", kind)
            m.set_position(positions - tokens)
            out[kind] = [m.prefill(ids)[0], m.read_hidden(0), m.read_hidden(1), *m.read_kv(1, positions - 1)]
        assert all(np.array_equal(a, b) for a, b in zip(out["1"], out["2"])) == (positions <= longest)
        assert all(rel_err(a, b) < 2e-3 for a, b in zip(out["1"], out["2"]))
    m.Dispose()


@pytest.mark.parametrize("at", [32, 33, 34, 300, 416])
def test_a_key_that_is_not_a_number(factory, monkeypatch, at):
    """Every exponential (positions 32, 33 and 416 go through the polynomial) passes a NaN on, as the warp-level kernel does."""
    cfg = synth.get_config("s3", gain_std=0.1)
    m = create_synthetic_model(cfg, 640, factory=factory, kv_dtype="f16")
    rng = np.random.default_rng(at)
    k, v = (rng.standard_normal((600, cfg.kvDim), dtype=np.float32) for _ in "kv")
    k[at, :cfg.d] = np.nan
    m.write_kv_range(0, 0, k, v)
    ids = synth.prompt_ids(cfg, 33, 8)
    out = {}
    for kind in ("1", "2"):
        monkeypatch.setenv("NFAI_PREFILL_ATTN", kind)
        m.set_position(500)
        m.prefill(ids)
        out[kind] = [m.read_hidden(1)] + [a for p in (500, 532) for a in m.read_kv(1, p)]
    m.Dispose()
    for a, b in zip(out["1"], out["2"]):
        assert np.isnan(a).all() and np.isnan(b).all()


def test_keys_beyond_float16(factory, monkeypatch):
    """Every key's last component is -infinity in the cache and every query's is positive: all scores of a row are -infinity, and 0 / 0
    is not a number in either kernel."""
    cfg = synth.get_config("s3")
    plain = synth.gen_tensor

    def gen_tensor(cfg, name, *args):
        w = plain(cfg, name, *args)
        if name == "token_embd.weight":
            w[:, 0] = 5.0  # (22 after the norm)
        if name in ("blk.0.attn_q.weight", "blk.0.attn_k.weight"):
            rows = [63] if "_k" in name else [63, 127, 191, 255]  # of the first KV group
            w[rows] = 0
            w[rows, 0] = -60000.0 if "_k" in name else 1.0
        return w
    monkeypatch.setattr(synth, "gen_tensor", gen_tensor)
    metadata = dict(synth.metadata(cfg), **{"llama.rope.dimension_count": 32})  # (the last components are not rotated)
    m = LlamaModel(factory.ctx, metadata, synthetic_tensors(cfg), 512, kv_dtype="f16")
    ids = synth.prompt_ids(cfg, 400, 10)
    for kind in ("1", "2"):
        monkeypatch.setenv("NFAI_PREFILL_ATTN", kind)
        m.reset()
        m.prefill(ids)
        k, _ = m.read_kv(0, 399)
        assert k[63] == -np.inf and np.isfinite(np.delete(k, 63)).all()
        assert np.isnan(m.read_hidden(0)).all(), kind
    m.Dispose()


@pytest.mark.parametrize("key,tokens", [("s1", 1601), ("s2", 300), ("s1", 37)])
def test_repeated_prompts_agree_to_the_bit(factory, key, tokens):
    """Kernels of every kind right behind one another (the next one's set-up runs beside the last one's end): what one leaves in
    flight would show in another's barriers or tiles."""
    cfg = synth.get_config(key, gain_std=0.1)
    m = create_synthetic_model(cfg, tokens, factory=factory)
    ids = synth.prompt_ids(cfg, tokens, 3)
    first = None
    for _ in range(8):
        m.reset()
        got = [m.prefill(ids)[0]] + [m.read_hidden(l) for l in range(cfg.L)] + [a for l in range(cfg.L) for a in m.read_kv(l, tokens // 2)]
        assert all(np.isfinite(a).all() for a in got)
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(got, first))
    m.Dispose()
