"""The dense GEMMs at the edges of a pair of CTAs' tile: 256 channels, 84 rows (W8A8: 256), columns of the digit operand in
steps of 32, k cut over the pairs of a cluster, several tiles per pair, and outputs whose rows are not aligned."""
import ctypes as C

import numpy as np
import pytest

from buddy_mlir_b200 import _lib

pytestmark = pytest.mark.gpu


def call(op, A, Q, s, ldc=0, bias=None, residual=None, silu=False):
    """C[:, :N] of a call whose output rows are ldc apart; what lies between them stays as it was."""
    import torch
    from gpu_util import dev, packed_weight, ptr, stream
    lib = _lib.load()
    (M, K), N = A.shape, Q.shape[1]
    w = packed_weight(_lib.W_I8, Q, K, N)
    ds, dA = dev(s), dev(A)
    db, dr = (None if v is None else dev(v) for v in (bias, residual))
    cols = N // 2 if silu else N
    ldc = ldc or cols
    out = torch.full((M, ldc), 7.0, device="cuda")
    weight = _lib.Weight(_lib.W_I8, 0, K, N, ptr(w), ptr(ds), _lib.F32, 0, None if db is None else ptr(db))
    bytes_of = lib.b200_gemm_w8_workspace_bytes if op == "w8" else lib.b200_gemm_w8a8_workspace_bytes
    ws = torch.zeros(bytes_of(M, K), dtype=torch.uint8, device="cuda")
    if op == "w8":
        _lib.check(lib.b200_gemm_w8(C.byref(weight), ptr(dA), M, K, ptr(out), ldc, None if dr is None else ptr(dr), N, None, 0.0, int(silu), ptr(ws), ws.numel(), stream()))
    else:
        _lib.check(lib.b200_gemm_w8a8(C.byref(weight), ptr(dA), M, K, ptr(out), ldc, ptr(ws), ws.numel(), stream()))
    _lib.check(lib.b200_gemm_w8_status(ptr(ws), stream()))
    out = out.cpu().numpy()
    assert (out[:, cols:] == 7.0).all()
    return out[:, :cols]


def inputs(M, N, K, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((M, K)).astype(np.float32), rng.integers(-128, 128, (K, N)).astype(np.int8),
            rng.uniform(0.001, 0.01, N).astype(np.float32), rng)


# one tile, two, and several turns of the 74 pairs; k whole, and in two and four shares whose rows do not divide
@pytest.mark.parametrize("M,N,K", [(2, 256, 64), (3, 257, 8960), (5, 255, 1600), (16, 513, 640), (17, 128, 4160), (83, 300, 8960), (84, 256, 1536),
                                   (86, 1000, 512), (168, 1536, 1024), (169, 511, 2048), (250, 20001, 64), (2048, 900, 192)])
def test_pair_edges(M, N, K):
    A, Q, s, rng = inputs(M, N, K, M + N + K)
    b, res = rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
    want = (A.astype(np.float64) @ Q.astype(np.float64)) * s + b + res
    got = call("w8", A, Q, s, ldc=N + 3, bias=b, residual=res)
    # 2^-23 of a row's largest activation in every product, f32 roundings of the digits' sums
    assert np.abs(got - want).max() / np.abs(want).max() < 4e-6


@pytest.mark.parametrize("M,N,K", [(1, 258, 64), (7, 512, 8960), (43, 18000, 128), (85, 270, 1536)])
def test_gate_up_pairs(M, N, K):
    A, Q, s, _ = inputs(M, N, K, M + N)
    A[0] *= 40.0                  # gates far below and above zero: e^-g overflows, and 1 / (1 + e^-g) is one
    y = (A.astype(np.float64) @ Q.astype(np.float64)) * s
    g, u = y[:, 0::2], y[:, 1::2]
    with np.errstate(over="ignore"):
        want = g / (1.0 + np.exp(-g)) * u
    got = call("w8", A, Q, s, silu=True)
    assert (np.abs(got - want).max(1) / np.abs(want).max(1)).max() < 1e-5


# integer sums: bit-identical to one product over the whole of k, however it is cut
@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (31, 257, 8960), (33, 1536, 4096), (255, 300, 1600), (256, 512, 640), (257, 255, 8960), (700, 9001, 192)])
def test_w8a8_pair_edges(M, N, K):
    A, Q, s, _ = inputs(M, N, K, M * 3 + N)
    scale = np.maximum(np.float32(np.abs(A).max()) * (np.float32(1) / np.float32(127)), np.float32(1e-10))
    q = np.clip(np.rint(A * (np.float32(1) / scale)), -128, 127)
    want = (q @ Q.astype(np.float64)).astype(np.float32) * (scale * s)
    assert np.array_equal(call("w8a8", A, Q, s, ldc=N + 1), want)


# k in three shares: of one row, of rows and blocks of k that three does not divide, and of rows of which a share is empty
@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (2, 4090, 3200), (24, 4096, 4160), (64, 4000, 6016), (200, 1536, 8960)])
def test_three_shares(M, N, K):
    A, Q, s, rng = inputs(M, N, K, M + K)
    if M > 2:
        A[M // 2, K // 2] *= 3000
    res = rng.standard_normal((M, N)).astype(np.float32)
    want = (A.astype(np.float64) @ Q.astype(np.float64)) * s + res
    got = call("w8", A, Q, s, residual=res)
    # as above, row by row: one row is far larger than the others
    assert (np.abs(got - want).max(1) / np.abs(want).max(1)).max() < 4e-6


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (25, 4090, 4160), (301, 1536, 8960)])
def test_w8a8_three_shares(M, N, K):
    A, Q, s, _ = inputs(M, N, K, M * 3 + K)
    scale = np.maximum(np.float32(np.abs(A).max()) * (np.float32(1) / np.float32(127)), np.float32(1e-10))
    q = np.clip(np.rint(A * (np.float32(1) / scale)), -128, 127)
    assert np.array_equal(call("w8a8", A, Q, s), (q @ Q.astype(np.float64)).astype(np.float32) * (scale * s))


# a row of six digits in one row tile of several, one turn of the pairs and several: the rows beside it are what they are without it
@pytest.mark.parametrize("M,N,K,silu", [(90, 1000, 512, False), (170, 12000, 640, False), (333, 18000, 256, True), (700, 1536, 1088, False), (1000, 2048, 256, True)])
def test_narrow_tiles_after_a_wide_one(M, N, K, silu):
    A, Q, s, rng = inputs(M, N, K, M + N)
    res = None if silu else rng.standard_normal((M, N)).astype(np.float32)
    narrow = call("w8", A, Q, s, residual=res, silu=silu)
    row = M // 2
    A[row, 5] *= 3000
    got = call("w8", A, Q, s, residual=res, silu=silu)
    others = np.arange(M) != row
    assert np.array_equal(got[others], narrow[others])
    y = (A[row].astype(np.float64) @ Q.astype(np.float64)) * s
    with np.errstate(over="ignore"):
        want = y[0::2] / (1.0 + np.exp(-y[0::2])) * y[1::2] if silu else y + res[row]
    assert np.abs(got[row] - want).max() / np.abs(want).max() < (1e-5 if silu else 4e-6)
