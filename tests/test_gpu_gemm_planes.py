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


def columns_off(y, A, Q, s):
    """Largest error of each column of y against f64, over the column's own rms (the rows have the same distribution)."""
    want = (A.astype(np.float64) @ Q.astype(np.float64)) * s
    return np.abs(y - want).max(0) / np.sqrt((want ** 2).mean(0))


@pytest.mark.parametrize("M,N,K", [(24, 130, 8960), (43, 256, 1536), (64, 1536, 320), (300, 20000, 192)])
@pytest.mark.parametrize("times", [1, 20, 100, 1000, 10000, 1e8])
def test_rows_with_one_large_channel(M, N, K, times):
    """Columns that do not use the channel keep the precision of the rest: an element's rounding is at most 2^-19 of the rest's rms
    (as two bf16 terms leave it), and the largest of about 10^6 sums of such errors lies near 5 of their rms."""
    from gpu_util import dev, gemm_w8, packed_weight
    rng = np.random.default_rng(M + N)
    A = rng.standard_normal((M, K)).astype(np.float32)
    A[:, 17] *= np.float32(times)
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    Q[17, ::2] = 0
    s = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y = gemm_w8(packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(A)).cpu().numpy()
    assert columns_off(y, A, Q, s).max() < 2e-5


@pytest.mark.parametrize("M", [1, 20, 21, 22, 42, 64, 85, 127])
@pytest.mark.parametrize("N,K", [(70, 4160), (20000, 192), (512, 1536)])
def test_wide_rows_among_others(M, N, K):
    """Every third row has outliers, so that passes with and without such rows meet in a tile; residual added in place, and a row
    does not depend on its neighbours."""
    from gpu_util import dev, gemm_w8, packed_weight
    rng = np.random.default_rng(M + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    A[::3, 5] = 3.7e4
    A[::3, 9] = -12345.678
    A[M // 2:M // 2 + 1] *= np.float32(1e-39)     # subnormal
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    Q[[5, 9], ::2] = 0
    s = rng.uniform(0.001, 0.01, N).astype(np.float32)
    w, ds = packed_weight(_lib.W_I8, Q, K, N), dev(s)
    y = gemm_w8(w, ds, K, N, dev(A)).cpu().numpy()
    want = (A.astype(np.float64) @ Q.astype(np.float64)) * s
    scale = np.sqrt((want ** 2).reshape(M, N // 2, 2).mean(1))   # of the row's columns without, and with the channels
    off = np.abs(y - want).reshape(M, N // 2, 2) / np.maximum(scale[:, None], 1e-44)
    ok = np.arange(M) != M // 2
    assert not ok.any() or off[ok].max() < 2e-5
    assert off[~ok].max() < 2e-5 or np.abs(y - want)[~ok].max() < 1e-44    # (results are subnormal too)
    for m in sorted({0, M - 1, M // 3 * 3 if M // 3 * 3 < M else 0}):
        assert np.array_equal(gemm_w8(w, ds, K, N, dev(A[m:m + 1].copy())).cpu().numpy()[0], y[m]) or N < 128 * 148
    res = rng.standard_normal((M, N)).astype(np.float32)
    assert np.array_equal(gemm_w8(w, ds, K, N, dev(A), residual=dev(res)).cpu().numpy(), res + y)


def test_rows_of_few_values_and_without_finite_scale():
    from gpu_util import dev, gemm_w8, packed_weight
    rng = np.random.default_rng(1)
    M, N, K = 48, 256, 512
    A = np.zeros((M, K), np.float32)
    A[:, 3] = np.float32(3.0)             # one value in a row of zeros is exact
    A[5] = rng.standard_normal(K) * 1e-30
    A[5, 0] = 3e38                        # the others lie 2^-227 below it: six digits reach 2^-45, so its column decides
    A[6, 1], A[7, 2] = np.nan, -np.inf
    A[8] = np.float32(1.9921874)          # at the largest mantissas that three digits hold
    A[9] = np.float32(-1.9999999)
    A[10] = np.where(np.arange(K) % 2, 1.9921875, -1.984375)
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    Q[0] = np.where(Q[0] == 0, 1, Q[0])
    s = np.ones(N, np.float32)
    y = gemm_w8(packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(A)).cpu().numpy()
    with np.errstate(invalid="ignore"):
        want = A.astype(np.float64) @ Q.astype(np.float64)
    for m in range(M):
        if m in (6, 7):
            assert not np.isfinite(y[m]).any()
        elif m == 5:
            with np.errstate(over="ignore"):
                np.testing.assert_allclose(y[m], want[m].astype(np.float32), rtol=1e-6, atol=0)
        elif m in (8, 9, 10):
            assert np.abs(y[m] - want[m]).max() / np.abs(want[m]).max() < 1e-6
        else:
            assert np.array_equal(y[m], want[m])
