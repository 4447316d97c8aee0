"""Tiles of the prompt kernels at their edges: products over pairs of SMs, against float64 products of the same operands."""
import numpy as np
import pytest

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
