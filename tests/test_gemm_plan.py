"""How the dense GEMM is laid over the chip, over the stand-in runtime: shares of k only while all of their clusters run at once (one
more than the chip holds takes a second turn, which costs more than the shares give)."""
import ctypes as C

import numpy as np

import fake_runtime

HELD = {2: 33, 3: 22, 4: 15}   # clusters of 2 x shares CTAs, as the stand-in answers


class Params(C.Structure):
    _fields_ = [("M", C.c_int), ("N", C.c_int), ("K", C.c_int), ("pointers", C.c_void_p * 5), ("strides", C.c_int64 * 2), ("silu_pairs", C.c_int),
                ("splits", C.c_int), ("share_rows", C.c_int), ("tiles", C.c_int), ("m_tiles", C.c_int)]


def test_clusters_run_at_once(tmp_path):
    fake_runtime.run(tmp_path, "test_gemm_plan", "plans")


def plans(fake):
    from buddy_mlir_b200 import _lib
    lib, seen = _lib.load(), []

    def launch(name, grid, args):
        if "gemm_i8_kernel" in name:
            p = C.cast(args[2], C.POINTER(Params))[0]
            seen.append((p.M, p.N, p.K, p.splits, p.share_rows, p.tiles, p.m_tiles, grid[0]))
    fake.on_launch(launch)
    buf = np.zeros(1 << 22, dtype=np.uint8)
    at = (buf.ctypes.data + 255) // 256 * 256
    taken = set()
    for N, K in ((4096, 12288), (4096, 4096), (1536, 8960), (500, 8960), (3000, 6016), (1000, 4096), (17920, 1536), (64, 64), (300, 192), (20001, 512)):
        w = _lib.Weight(_lib.W_I8, 0, K, N, at, at, _lib.F32, 0, None)
        for M in (1, 2, 5, 17, 24, 33, 64, 84, 85, 100, 200, 255, 256, 257, 366, 512, 700, 1024, 2048, 5000):
            _lib.check(lib.b200_gemm_w8(C.byref(w), at, M, K, at, N, None, 0, None, 0.0, 0, at, 1 << 40, None))
            _lib.check(lib.b200_gemm_w8a8(C.byref(w), at, M, K, at, N, at, 1 << 40, None))
            for call in seen:
                m, n, k, splits, share_rows, tiles, m_tiles, ctas = call
                rows = -(-M // m_tiles)
                assert (m, n, k) == (M, N, K) and tiles == m_tiles * -(-N // 256) and share_rows * splits >= rows, call
                if splits == 1:
                    assert ctas == 2 * min(tiles, 74), call
                else:
                    assert ctas == 2 * splits * tiles and tiles <= HELD[splits] and splits <= -(-K // 128) // 2, call
                taken.add(splits)
            del seen[:]
    assert taken == {1, 2, 3, 4}
