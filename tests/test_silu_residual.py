"""b200_gemm_w8 with SiLU pairs and a residual, which has the output's N / 2 columns and counts for nothing: the kernel, which asks for
residual rows of N columns a tile ahead, must not be given it (over the stand-in runtime: reading it would be out of range)."""
import ctypes as C

import numpy as np

import fake_runtime


class Params(C.Structure):   # the head of the kernel's parameters
    _fields_ = [("M", C.c_int), ("N", C.c_int), ("K", C.c_int), ("scale", C.c_void_p), ("bias", C.c_void_p), ("row_scale", C.c_void_p),
                ("residual", C.c_void_p), ("C", C.c_void_p)]


def test_the_kernel_gets_no_residual_with_silu_pairs(tmp_path):
    fake_runtime.run(tmp_path, "test_silu_residual", "residual_of_calls")


def residual_of_calls(fake):
    from buddy_mlir_b200 import _lib
    lib, seen = _lib.load(), []

    def launch(name, grid, args):
        if "gemm_i8_kernel" in name:
            p = C.cast(args[2], C.POINTER(Params))[0]
            seen.append((p.M, p.N, p.K, p.C, p.residual))
    fake.on_launch(launch)
    buf = np.zeros(1 << 22, dtype=np.uint8)
    at = (buf.ctypes.data + 255) // 256 * 256
    for M, K in ((4, 128), (24, 8960), (200, 512)):
        w = _lib.Weight(_lib.W_I8, 0, K, 64, at, at, _lib.F32, 0, None)
        for residual, silu, want in ((None, 0, None), (at + 4096, 0, at + 4096), (None, 1, None), (at + 4096, 1, None)):
            _lib.check(lib.b200_gemm_w8(C.byref(w), at, M, K, at + 256, 64 >> silu, residual, 64 >> silu, None, 0.0, silu, at, 1 << 40, None))
            assert seen.pop() == (M, 64, K, at + 256, want) and not seen
