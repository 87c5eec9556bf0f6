"""Which kernel takes one row over few weights: the integer tensor cores, or the CUDA cores (on the host: the choice needs no GPU)."""
import ctypes as C

from buddy_mlir_b200 import _lib


def tensor_cores(kind, N, K, group=0, x=_lib.F32, M=1):
    f = _lib.load()["_ZN4b20014gemv_mma_takesEPK11b200_weightPK14b200_gemv_args"]
    f.restype = C.c_bool
    w = _lib.Weight(kind, group, K, N, 1 << 20, 1 << 20, _lib.F32 if kind == _lib.W_I8 else _lib.F16, 0, None)
    return f(C.byref(w), C.byref(_lib.GemvArgs(1 << 20, x, _lib.F32, K, N, 1 << 20, None, None, 0.0, M, 0, 0)))


def test_int4_rows_that_the_cuda_cores_finish_sooner():
    """Per channel, and whole blocks in groups, up to five blocks of 1024: from memory and from L2 alike."""
    for N in (64, 500, 1024, 2048):
        for x in (_lib.F32, _lib.F16, _lib.BF16):
            for K in (2560, 2816, 3584, 5120):
                assert not tensor_cores(_lib.W_U4, N, K, x=x), (N, K, x)
        assert not tensor_cores(_lib.W_U4, N, 5120, 128)
    assert not tensor_cores(_lib.W_U4, 2048, 3072) and not tensor_cores(_lib.W_U4, 500, 3072, x=_lib.BF16) and not tensor_cores(_lib.W_U4, 500, 4096) and not tensor_cores(_lib.W_U4, 500, 4096, 128)


def test_rows_that_go_to_the_tensor_cores():
    for N in (64, 500, 1024):
        for x in (_lib.F32, _lib.F16, _lib.BF16):
            for K in (6144, 8960, 14336):
                assert tensor_cores(_lib.W_U4, N, K, x=x) and tensor_cores(_lib.W_U4, N, K, 128, x) and tensor_cores(_lib.W_I8, N, K, x=x)
            assert tensor_cores(_lib.W_U4, N, 2560, 128, x) and tensor_cores(_lib.W_U4, N, 3584, 128, x) and tensor_cores(_lib.W_I8, N, 2560, x=x)
        assert tensor_cores(_lib.W_U4, N, 4096, x=_lib.F16) and tensor_cores(_lib.W_U4, N, 4096, 128, _lib.BF16)
    assert tensor_cores(_lib.W_U4, 1536, 4096) and tensor_cores(_lib.W_U4, 2500, 5120) and tensor_cores(_lib.W_U4, 500, 2560, M=2)
    assert tensor_cores(_lib.W_I8, 5000, 1536) and not tensor_cores(_lib.W_I8, 1536, 1536) and not tensor_cores(_lib.W_U4, 1536, 1536, 128)
