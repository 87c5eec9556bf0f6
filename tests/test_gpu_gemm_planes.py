"""b200_gemm_w8 at the edges of its tiles: 42 activation rows per tile, 128 / 256 columns, 128-byte k blocks (the last one
half), k ranges split over CTAs, and rows of very different magnitude (every row has a fixed-point scale of its own)."""
import numpy as np
import pytest

import oracle_lib as orc
from buddy_mlir_b200 import _lib

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a.astype(np.float64) - b.astype(np.float64)).max() / np.abs(b.astype(np.float64)).max())


@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (41, 130, 192), (42, 127, 128), (43, 129, 320), (84, 250, 4160), (85, 70, 8960),
                                   (127, 256, 1536), (300, 9001, 192), (1500, 3000, 64), (33, 20000, 576)])
def test_tile_edges(M, N, K):
    from gpu_util import dev, gemm_w8, packed_weight
    rng = np.random.default_rng(M * 3 + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    Q = rng.integers(-128, 128, (K, N)).astype(np.int8)
    s = rng.uniform(0.001, 0.01, N).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    y = gemm_w8(packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(A), residual=dev(res)).cpu().numpy()
    want = (A.astype(np.float64) @ Q.astype(np.float64)) * s + res
    assert rel(y, want) < 4e-6


def test_rows_keep_their_own_scale():
    from gpu_util import dev, gemm_w8, packed_weight
    rng = np.random.default_rng(8)
    M, N, K = 50, 140, 1536
    A = (rng.standard_normal((M, K)) * np.logspace(-20, 15, M)[:, None]).astype(np.float32)
    A[7] = 0
    A[9, 3] = np.inf
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    s = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y = gemm_w8(packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(A)).cpu().numpy()
    for m in range(M):
        if m == 9:
            assert not np.isfinite(y[m]).any()
        elif m == 7:
            assert (y[m] == 0).all()
        else:
            assert rel(y[m], orc.gemm_w8_prefill_f32(A[m:m + 1], Q, s, np.zeros((1, N), np.float32))[0]) < 4e-6
