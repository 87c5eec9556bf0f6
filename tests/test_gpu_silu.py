"""SiLU pairs folded into a projection's store are the bits of the projection and the separate operation after it, whatever the
range of the gates: the dense GEMM against itself and b200_silu_mul, and the two int8 forms of one row against each other."""
import ctypes as C

import numpy as np
import pytest

from buddy_mlir_b200 import _lib

pytestmark = pytest.mark.gpu


def weight(K, N, seed):
    from gpu_util import dev, packed_weight
    rng = np.random.default_rng(seed)
    Q, s = rng.integers(-127, 128, (K, N)).astype(np.int8), rng.uniform(0.5, 1.5, N).astype(np.float32) / np.float32(40 * np.sqrt(K))
    keep = packed_weight(_lib.W_I8, Q, K, N), dev(s)
    return _lib.Weight(_lib.W_I8, 0, K, N, keep[0].data_ptr(), keep[1].data_ptr(), _lib.F32, 0, None), keep, rng


def silu_mul(y):
    import torch
    from gpu_util import ptr, stream
    g, u = y[:, 0::2].contiguous(), y[:, 1::2].contiguous()
    out = torch.empty_like(g)
    _lib.check(_lib.load().b200_silu_mul(ptr(g), ptr(u), ptr(out), C.c_int64(g.numel()), stream()))
    return out.cpu().numpy()


def same(a, b):
    return np.array_equal(a.view(np.int32), b.view(np.int32))


# k in shares and whole, one turn of the pairs and several; rows from tiny gates to gates whose e^-g overflows
@pytest.mark.parametrize("M,N,K,wide", [(7, 512, 8960, False), (84, 258, 512, True), (333, 4096, 1536, True), (1024, 17920, 512, False)])
def test_dense_gemm(M, N, K, wide):
    import torch
    from gpu_util import dev, ptr, stream
    lib = _lib.load()
    w, keep, rng = weight(K, N, M + N)
    A = rng.standard_normal((M, K)).astype(np.float32) * np.float32(10) ** np.linspace(-3, 2, M, dtype=np.float32)[:, None]
    if wide:                     # a row of six digits
        A[M // 2, 17] *= 3000
    dA, ws = dev(A), torch.zeros(lib.b200_gemm_w8_workspace_bytes(M, K), dtype=torch.uint8, device="cuda")
    out = []
    for silu in (0, 1):
        y = torch.empty(M, N >> silu, device="cuda")
        _lib.check(lib.b200_gemm_w8(C.byref(w), ptr(dA), M, K, ptr(y), N >> silu, None, 0, None, 0.0, silu, ptr(ws), ws.numel(), stream()))
        _lib.check(lib.b200_gemm_w8_status(ptr(ws), stream()))
        out.append(y)
    assert out[0].abs().max() > 100
    assert same(out[1].cpu().numpy(), silu_mul(out[0]))


@pytest.mark.parametrize("N,K,size", [(512, 1536, 1.0), (4098, 512, 30.0), (17920, 1536, 1e-3), (256, 4096, 100.0)])
def test_int8_forms_of_one_row(N, K, size):
    """Both are reached through a w8a8 session only: called here by their symbols."""
    import torch
    from gpu_util import dev, ptr, stream
    lib = _lib.load()
    row_form = lib["_ZN4b20020gemv_i8_fused_launchEPK11b200_weightPKfS4_fS4_PfiP11CUstream_st"]
    rows_form = lib["_ZN4b20015gemm_w8a8_fusedEPK11b200_weightPKfilPflS4_liPvlbP11CUstream_st"]
    w, keep, rng = weight(K, N, N)
    dA = dev((rng.standard_normal((1, K)) * size).astype(np.float32))
    ws = torch.zeros(lib.b200_gemm_w8a8_workspace_bytes(1, K), dtype=torch.uint8, device="cuda")
    i64, f32, silu = C.c_int64, C.c_float, 1
    one, dense, plain = (torch.empty(1, n, device="cuda") for n in (N // 2, N // 2, N))
    _lib.check(row_form(C.byref(w), ptr(dA), None, f32(0), None, ptr(one), silu, stream()))
    _lib.check(rows_form(C.byref(w), ptr(dA), 1, i64(K), ptr(dense), i64(N // 2), None, i64(0), silu, ptr(ws), i64(ws.numel()), C.c_bool(False), stream()))
    _lib.check(lib.b200_gemm_w8a8(C.byref(w), ptr(dA), 1, K, ptr(plain), N, ptr(ws), ws.numel(), stream()))
    torch.cuda.synchronize()
    assert same(one.cpu().numpy(), dense.cpu().numpy())
    assert same(dense.cpu().numpy(), silu_mul(plain))


# one turn of the pairs, k in shares, wide rows: the three places that ask for residual rows
@pytest.mark.parametrize("M,N,K,wide", [(100, 512, 512, False), (24, 256, 8960, False), (84, 514, 512, True)])
def test_a_residual_beside_silu_pairs_is_left_alone(M, N, K, wide):
    """b200_gemm_w8 has no residual for SiLU pairs: one that is given all the same, of the output's N / 2 columns, counts for nothing."""
    import torch
    from gpu_util import dev, ptr, stream
    lib = _lib.load()
    w, keep, rng = weight(K, N, M)
    A = rng.standard_normal((M, K)).astype(np.float32)
    if wide:
        A[M // 2, 17] *= 3000
    dA, ws = dev(A), torch.zeros(lib.b200_gemm_w8_workspace_bytes(M, K), dtype=torch.uint8, device="cuda")
    res, out = torch.full((M, N // 2), float("nan"), device="cuda"), []
    for r in (None, ptr(res)):
        y = torch.empty(M, N // 2, device="cuda")
        _lib.check(lib.b200_gemm_w8(C.byref(w), ptr(dA), M, K, ptr(y), N // 2, r, N // 2, None, 0.0, 1, ptr(ws), ws.numel(), stream()))
        _lib.check(lib.b200_gemm_w8_status(ptr(ws), stream()))
        out.append(y.cpu().numpy())
    assert same(*out)
