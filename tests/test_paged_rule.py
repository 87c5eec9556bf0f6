"""When a decode step's attention is one kernel (a cluster of up to eight CTAs per row and kv head), and when the general kernels take it:
a CTA's range of keys is a chain, and few rows of long contexts leave it long while most of the chip is idle."""
import ctypes as C

from buddy_mlir_b200 import _lib


def takes(rows, q_heads, kv_heads, D, longest, qkv=1 << 20, ld=None, pool=1 << 20):
    f = _lib.load()["_ZN4b20018paged_decode_takesEPKflS1_S1_iiiii"]
    f.restype = C.c_bool
    return f(C.c_void_p(qkv), C.c_int64(ld or (q_heads + 2 * kv_heads) * D), C.c_void_p(pool), C.c_void_p(pool), q_heads, kv_heads, D, rows, longest)


def test_ranges_that_pay():
    for rows, longest in ((1, 8000), (2, 8000), (4, 8000)):
        assert not takes(rows, 12, 2, 128, longest)
    for rows, longest in ((1, 3000), (4, 4000), (8, 6000), (24, 700), (37, 2000), (74, 1024), (300, 1024)):
        assert takes(rows, 12, 2, 128, longest)
    for rows, longest in ((1, 4000), (2, 8000), (8, 4000), (16, 4000), (37, 2000)):
        assert not takes(rows, 8, 1, 128, longest)
    for rows, longest in ((1, 2000), (16, 2000), (24, 2500), (64, 4000), (128, 1000)):
        assert takes(rows, 8, 1, 128, longest)
    assert not takes(1, 32, 8, 128, 8192) and takes(2, 32, 8, 128, 8192) and takes(8, 32, 8, 128, 4096)


def test_what_the_kernel_is_built_for():
    assert takes(1, 8, 8, 64, 1) and takes(65535, 4, 2, 128, 1024)
    assert not takes(1, 8, 8, 32, 1) and not takes(1, 10, 2, 128, 1) and not takes(1, 14, 2, 128, 1) and not takes(65536, 4, 2, 128, 10)
    assert not takes(1, 4, 2, 128, 100, qkv=(1 << 20) + 4) and not takes(1, 4, 2, 128, 100, pool=(1 << 20) + 8) and not takes(1, 4, 2, 128, 100, ld=1026)
    for rows, longest in ((1, 8193), (19, 1025), (10, 2049)):
        assert not takes(rows, 32, 8, 128, longest)
