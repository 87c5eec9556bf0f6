"""b200_gemv on the integer tensor cores at the sizes where its tiling can go wrong: ragged rows, short last
blocks (int8: K % 512, int4: every K % 1024 that is a multiple of 128), every tile of activation rows, activation
slabs that do not fit shared memory at once, 16-bit activations, non-finite activations."""
import numpy as np
import pytest

import oracle_lib as orc
from buddy_mlir_b200 import _lib

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("M,N,K", [(2, 8, 64), (2, 1, 16), (3, 77, 528), (5, 1001, 1040), (8, 33, 5008), (12, 333, 8976),
                                   (16, 250, 12304), (1, 4099, 1552), (2, 50, 1001)])
def test_int8_edges(M, N, K):
    from gpu_util import dev, gemv, packed_weight
    rng = np.random.default_rng(M * 7 + N + K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    Q = rng.integers(-128, 128, (K, N)).astype(np.int8)
    s = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y = gemv(_lib.W_I8, packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(x)).cpu().numpy()
    assert rel(y, orc.gemv_w8_f32(x, Q, s)) < 1e-5


@pytest.mark.parametrize("M,N,K", [(2, 500, 128), (3, 66, 384), (2, 130, 640), (4, 34, 896), (5, 1000, 1152), (1, 9000, 1664),
                                   (7, 18, 1280), (10, 250, 1792), (16, 100, 9088), (16, 64, 2944)])
def test_int4_group128_edges(M, N, K):
    from gpu_util import dev, gemv, packed_scales, packed_weight
    rng = np.random.default_rng(M + N * 3 + K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    P = rng.integers(0, 256, (K, N // 2)).astype(np.uint8)
    s = rng.uniform(0.001, 0.01, (K // 128, N)).astype(np.float16)
    y = gemv(_lib.W_U4, packed_weight(_lib.W_U4, P, K, N, 0), packed_scales(s, _lib.F16, K // 128, N), K, N, dev(x),
             group=128, scale_dtype=_lib.F16).cpu().numpy()
    assert rel(y, orc.gemv_w4g_f32(x, P, s, 128)) < 1e-5


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("M", [2, 9])
def test_norm_silu_and_16_bit_rows(dtype, M):
    import torch
    from gpu_util import dev, gemv, packed_weight
    rng = np.random.default_rng(M)
    K, N = 1552, 2 * 77
    xt = torch.from_numpy((rng.standard_normal((M, K)) * 50).astype(np.float32)).to(
        torch.float16 if dtype == "f16" else torch.bfloat16).cuda()
    x = xt.float().cpu().numpy()
    nw = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    s = rng.uniform(0.0005, 0.001, N).astype(np.float32)
    y = gemv(_lib.W_I8, packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, xt, norm_w=dev(nw), silu=True,
             x_dtype=_lib.F16 if dtype == "f16" else _lib.BF16).cpu().numpy()
    for m in range(M):
        r = orc.gemv_w8_f32(orc.rmsnorm(x[m], nw, 1e-6)[None, :], Q, s)[0]
        assert rel(y[m], orc.silu_mul(np.ascontiguousarray(r[0::2]), np.ascontiguousarray(r[1::2]))) < 1e-5


def test_rows_of_very_different_size_and_a_row_with_a_nan():
    """Every activation row has a fixed-point scale of its own; a non-finite row yields no finite result."""
    from gpu_util import dev, gemv, packed_weight
    rng = np.random.default_rng(3)
    M, N, K = 4, 40, 1024
    x = rng.standard_normal((M, K)).astype(np.float32) * np.float32([[1e-30], [1e20], [1.0], [1.0]])
    x[2, 5] = np.nan
    x[3, :] = 0
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    s = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y = gemv(_lib.W_I8, packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(x)).cpu().numpy()
    ref = orc.gemv_w8_f32(x[[0, 1, 3]], Q, s)
    assert rel(y[0], ref[0]) < 1e-5 and rel(y[1], ref[1]) < 1e-5
    assert not np.isfinite(y[2]).any() and (y[3] == 0).all()


@pytest.mark.parametrize("times", [1, 200, 3000, 1e5, 1e9])
@pytest.mark.parametrize("kind,M,N,K", [("i8", 2, 77, 528), ("i8", 5, 1001, 1040), ("i8", 16, 250, 12304), ("i8", 1, 4100, 1552),
                                        ("u4", 2, 130, 640), ("u4", 5, 1000, 1152), ("u4", 1, 9000, 1664), ("u4", 16, 100, 9088),
                                        ("u4", 9, 40000, 2048)])
def test_rows_with_one_large_channel(kind, M, N, K, times):
    """Outputs that do not use the channel keep the precision of the rest: an element's rounding to four digits is at most 2^-22 of
    the rest; in f32 a lane adds up to K / 128 groups of four (96 here), sqrt(96 / 3) * 2^-24 = 3.4e-7 of the sum, which is up to 127 / 73
    of the column's size; the largest of 2000 such errors lies near 4.5 of their rms: 2.7e-6."""
    from gpu_util import dev, gemv, packed_scales, packed_weight
    rng = np.random.default_rng(M * 7 + N + K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[0 if M < 3 else slice(1, None, 2), 17] *= np.float32(times)     # some rows only
    if kind == "i8":
        Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
        Q[17, ::2] = 0
        s = rng.uniform(0.001, 0.01, N).astype(np.float32)
        y = gemv(_lib.W_I8, packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, dev(x)).cpu().numpy()
        want = (x.astype(np.float64) @ Q.astype(np.float64)) * s
    else:
        P = rng.integers(0, 256, (K, N // 2)).astype(np.uint8)
        P[17] = P[17] & 0xF0 | 8                                      # code 8 is zero; the low nibble is the even column
        s = rng.uniform(0.001, 0.01, (K // 128, N)).astype(np.float16)
        y = gemv(_lib.W_U4, packed_weight(_lib.W_U4, P, K, N, 0), packed_scales(s, _lib.F16, K // 128, N), K, N, dev(x),
                 group=128, scale_dtype=_lib.F16).cpu().numpy()
        q = np.stack([P & 15, P >> 4], axis=2).reshape(K, N).astype(np.float64) - 8
        want = x.astype(np.float64) @ (q * np.repeat(s.astype(np.float64), 128, axis=0))
    off = np.abs(y - want)
    for c in (0, 1):   # the columns without the channel, and with it, over their rms in each row
        size = np.sqrt((want[:, c::2] ** 2).mean(1, keepdims=True))
        assert (off[:, c::2] / size).max() < 4e-6


def test_wide_rows_norm_silu_accumulate_and_tiny_rows():
    from gpu_util import dev, gemv, packed_weight
    rng = np.random.default_rng(5)
    M, N, K = 6, 2 * 300, 1552
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[1, 40] = 3e5
    nw = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    Q = rng.integers(-127, 128, (K, N)).astype(np.int8)
    s = rng.uniform(0.0005, 0.001, N).astype(np.float32)
    w, ds = packed_weight(_lib.W_I8, Q, K, N), dev(s)
    y = gemv(_lib.W_I8, w, ds, K, N, dev(x), norm_w=dev(nw), silu=True).cpu().numpy()
    for m in range(M):
        r = orc.gemv_w8_f32(orc.rmsnorm(x[m], nw, 1e-6)[None, :], Q, s)[0]
        assert rel(y[m], orc.silu_mul(np.ascontiguousarray(r[0::2]), np.ascontiguousarray(r[1::2]))) < 1e-5
    y0 = rng.standard_normal((M, N)).astype(np.float32)
    y = gemv(_lib.W_I8, w, ds, K, N, dev(x), accumulate=True, y0=dev(y0.copy())).cpu().numpy()
    assert rel(y, y0 + orc.gemv_w8_f32(x, Q, s)) < 1e-5
    tiny = (x * np.float32(1e-36)).astype(np.float32)      # far below the smallest scale of four digits
    y = gemv(_lib.W_I8, w, ds, K, N, dev(tiny)).cpu().numpy()
    want = (tiny.astype(np.float64) @ Q.astype(np.float64)) * s
    for m in range(M):
        assert np.abs(y[m] - want[m]).max() / np.abs(want[m]).max() < 1e-5


@pytest.mark.parametrize("kind,M,N,K", [("u4", 3, 66, 1032), ("u4", 1, 20000, 2080), ("i8", 3, 55, 1001), ("i8", 7, 130, 8976)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_wide_rows_per_channel_and_odd_lengths(kind, M, N, K, dtype):
    import torch
    from gpu_util import dev, gemv, packed_scales, packed_weight
    rng = np.random.default_rng(M + K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[M // 2, K - 3] = 2e5
    xt = torch.from_numpy(x).cuda() if dtype == "f32" else torch.from_numpy(x).to(torch.bfloat16).cuda()
    x = xt.float().cpu().numpy()
    res = rng.standard_normal((M, N)).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    code = _lib.F32 if dtype == "f32" else _lib.BF16
    if kind == "i8":
        Q = rng.integers(-128, 128, (K, N)).astype(np.int8)
        s = rng.uniform(0.001, 0.01, N).astype(np.float32)
        y = gemv(_lib.W_I8, packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, xt, bias=dev(bias), residual=dev(res), x_dtype=code)
        q = Q.astype(np.float64)
    else:
        P = rng.integers(0, 256, (K, N // 2)).astype(np.uint8)
        s = rng.uniform(0.001, 0.01, N).astype(np.float16)
        y = gemv(_lib.W_U4, packed_weight(_lib.W_U4, P, K, N, 0), packed_scales(s.reshape(1, N), _lib.F16, 1, N), K, N, xt, scale_dtype=_lib.F16,
                 bias=dev(bias), residual=dev(res), x_dtype=code)
        q = np.stack([P & 15, P >> 4], axis=2).reshape(K, N).astype(np.float64) - 8
    want = (x.astype(np.float64) @ q) * s.astype(np.float64) + bias + res
    y = y.cpu().numpy()
    for m in range(M):   # (every row on its own: only one has the large element)
        assert np.abs(y[m] - want[m]).max() / np.abs(want[m]).max() < 1e-5


@pytest.mark.parametrize("kind,N,K", [("i8", 1, 2560), ("i8", 3, 2561), ("i8", 70, 2559), ("i8", 129, 3056), ("i8", 17, 8960), ("i8", 9, 14336),
                                      ("i8", 5, 40000), ("i8", 4200, 1501), ("u4", 2, 2560), ("u4", 34, 4096), ("u4", 66, 2688), ("u4", 18, 9088),
                                      ("u4", 4, 14336), ("u4", 5000, 1280)])
@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
def test_one_row_on_both_sides_of_the_line(kind, N, K, dtype):
    """One row over few weights, at the lengths where the kernel changes: bias, residual and accumulation against f64."""
    import torch
    from gpu_util import dev, gemv, packed_scales, packed_weight
    rng = np.random.default_rng(N + K)
    xt = torch.from_numpy(rng.standard_normal((1, K)).astype(np.float32)).to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[dtype]).cuda()
    code = {"f32": _lib.F32, "f16": _lib.F16, "bf16": _lib.BF16}[dtype]
    bias, res = rng.standard_normal(N).astype(np.float32), rng.standard_normal((1, N)).astype(np.float32)
    if kind == "i8":
        Q = rng.integers(-128, 128, (K, N)).astype(np.int8)
        s = rng.uniform(0.001, 0.01, N).astype(np.float32)
        y = gemv(_lib.W_I8, packed_weight(_lib.W_I8, Q, K, N), dev(s), K, N, xt, bias=dev(bias), residual=dev(res), x_dtype=code)
        w = Q.astype(np.float64) * s
    else:
        P = rng.integers(0, 256, (K, N // 2)).astype(np.uint8)
        s = rng.uniform(0.001, 0.01, (K // 128, N)).astype(np.float16)
        y = gemv(_lib.W_U4, packed_weight(_lib.W_U4, P, K, N, 0), packed_scales(s, _lib.F16, K // 128, N), K, N, xt, group=128,
                 scale_dtype=_lib.F16, bias=dev(bias), residual=dev(res), x_dtype=code)
        w = (np.stack([P & 15, P >> 4], axis=2).reshape(K, N).astype(np.float64) - 8) * np.repeat(s.astype(np.float64), 128, axis=0)
    want = xt.double().cpu().numpy() @ w + bias + res
    # f32 sums of K products: sqrt(K) * 2^-24 of the largest at most, here 40000: 1.2e-5
    assert np.abs(y.cpu().numpy() - want).max() / max(np.abs(want).max(), 1.0) < 1.2e-5
