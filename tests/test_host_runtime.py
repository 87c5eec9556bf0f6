"""The host side of the library over the stand-in CUDA runtime (fake_cudart.c): failures that are made on the host."""
import ctypes as C

import numpy as np

import fake_runtime


def test_a_pass_keeps_the_error_of_any_of_its_gemms(tmp_path):
    fake_runtime.run(tmp_path, "test_host_runtime", "errors_of_a_pass")


def errors_of_a_pass(fake):
    """Every GEMM of a pass in turn 'gives up': the n-th launch writes the code a bounded wait leaves, and what the kernels around
    it clear is cleared.  The pass has to fail, and the pass after it to succeed."""
    from buddy_mlir_b200 import TINY_MEGA, _lib, synthetic
    from buddy_mlir_b200.session import BatchSession, ModelSession
    state = {"n": 0, "fail": -1}

    def launch(name, grid, args):
        p = lambda i, kind: C.cast(args[i], C.POINTER(kind))[0]
        if "planes_kernel" in name:
            clear, at = p(11, C.c_int), p(10, C.c_void_p)
            C.memset(at, 0, 4 * clear)
        elif "absmax_kernel" in name and p(6, C.c_void_p):
            C.memset(p(6, C.c_void_p), 0, 4)
        elif "gemm_i8_kernel" in name:
            if state["n"] == state["fail"]:
                # GemmParams::error
                C.cast(C.cast(args[2], C.POINTER(C.c_void_p))[12], C.POINTER(C.c_int))[0] = 702
            state["n"] += 1
    fake.on_launch(launch)
    _, views = synthetic.make_f32_blob(TINY_MEGA, 3)
    for int8 in (False, True):
        s = ModelSession(TINY_MEGA)
        s.load_tensors(views, quantize_to="w8")
        s.set_activation_int8(int8)
        batch = None if int8 else BatchSession(s, 2, 16, 16, 64)

        def one_pass(fail):
            state.update(n=0, fail=fail)
            try:
                if batch is None:
                    s.prefill_rows(np.arange(5), 0, all_rows=False)
                else:
                    q = batch.add()
                    try:
                        batch.prefill(q, np.arange(5))
                    finally:
                        batch.remove(q)
            except _lib.B200Error as e:
                assert "code 702" in str(e)
                return False
            return True
        assert one_pass(-1)
        gemms = state["n"]
        assert gemms == 4 * TINY_MEGA.n_layers + 1
        for i in range(gemms):
            assert not one_pass(i), i
            assert one_pass(-1), i


def test_shared_memory_limits_are_raised_on_every_device(tmp_path):
    fake_runtime.run(tmp_path, "test_host_runtime", "calls_on_several_devices")


def calls_on_several_devices(fake):
    """The calls that need more than 48 KB of shared memory, on one device after the other, and back: the limit belongs to the
    device that is current."""
    from buddy_mlir_b200 import _lib
    lib, device = _lib.load(), fake.value("fake_device", C.c_int)
    buf = np.zeros(1 << 16, dtype=np.uint8)
    at = (buf.ctypes.data + 255) // 256 * 256
    for d in (0, 1, 0, 5):
        device.value = d
        for kind, K, N, M in ((_lib.W_I8, 8960, 1536, 5), (_lib.W_I8, 8960, 1536, 1), (_lib.W_U4, 4096, 14336, 16), (_lib.W_F32, 14336, 1024, 1),
                              (_lib.W_F32, 8960, 1536, 16), (_lib.W_I8, 70000, 1024, 4)):
            w = _lib.Weight(kind, 128 if kind == _lib.W_U4 else 0, K, N, at, at, _lib.F16 if kind == _lib.W_U4 else _lib.F32, 0, None)
            a = _lib.GemvArgs(at, _lib.F32, _lib.F32, K, N, at, None, None, 0.0, M, 0, 0)
            assert lib.b200_gemv(C.byref(w), C.byref(a), None) == 0, (d, kind, K, N, M, lib.b200_last_error())
        w = _lib.Weight(_lib.W_I8, 0, 1536, 1536, at, at, _lib.F32, 0, None)
        assert lib.b200_gemm_w8(C.byref(w), at, 64, 1536, at, 1536, None, 0, None, 0.0, 0, at, 1 << 40, None) == 0


def test_sessions_that_fit_without_the_decode_kernels_copy_of_the_weights(tmp_path):
    fake_runtime.run(tmp_path, "test_host_runtime", "sessions_in_little_memory")


def sessions_in_little_memory(fake):
    """The persistent decode kernel keeps the linear weights a second time.  Where there is no room for that, a session that runs
    without it still loads, prefills, serves batches and decodes."""
    import os
    from buddy_mlir_b200 import TINY_MEGA, _lib, synthetic
    from buddy_mlir_b200.session import BatchSession, ModelSession
    memory, used, peak = (fake.value("fake_" + n) for n in ("memory", "used", "peak"))
    cfg = TINY_MEGA.with_(max_len=64)
    _, views = synthetic.make_f32_blob(cfg, 3)

    def session(quantize=None):
        s = ModelSession(cfg)
        s.load_tensors(views, quantize_to=quantize)
        return s
    os.environ["BUDDY_B200_DECODE"] = "graph"
    s = session()
    plain_peak, plain = peak.value, used.value
    s.prefill_rows(np.arange(40), 0, all_rows=False)
    batch = BatchSession(s, 2, 16, 8, 64)
    busy_peak = peak.value
    batch.close()
    s.close()
    del os.environ["BUDDY_B200_DECODE"]
    s = session()
    assert s.uses_persistent_kernel() and used.value > 1.5 * plain
    full = used.value
    s.close()
    assert used.value == 0
    # no room for the copy when the model is finalised
    memory.value = max(plain_peak, busy_peak)
    s = session()
    assert not s.uses_persistent_kernel()
    s.decode(3)
    s.close()
    # room for it then, but not for what a prefill or a batch needs later
    for later in (lambda s: s.prefill_rows(np.arange(40), 0, all_rows=False), lambda s: BatchSession(s, 2, 16, 8, 64).close()):
        memory.value = 1 << 40
        s = session()
        memory.value = max(full, busy_peak)
        assert s.uses_persistent_kernel()
        later(s)
        assert not s.uses_persistent_kernel()
        s.position_ = 0
        s.decode(3)
        s.generate(3, 2)
        s.close()
    # pools that never fit do not cost the session its kernel: nothing, one and several of the pools go through
    for pages in (1 << 20, 2900, 900):
        memory.value = 1 << 40
        s = session()
        memory.value = full + 1000000
        try:
            BatchSession(s, 2, 16, pages, 64)
            raise SystemExit("the pools fit")
        except _lib.B200Error as e:
            assert "memory" in str(e)
        assert s.uses_persistent_kernel() and used.value == full
        s.decode(3)
        s.close()
    # the w8a8 arithmetic decodes without the kernel: no copy, until it is switched off
    memory.value = 1 << 40
    s = ModelSession(cfg)
    floats, ints = synthetic.split_w8a32(cfg, views, lambda w: (np.ones_like(w, dtype=np.int8), np.ones((1, w.shape[1]), np.float32)))
    s.load_blobs("w8a8", floats, ints)
    assert not s.uses_persistent_kernel()
    s.decode(3)
    s.set_activation_int8(False)
    assert s.uses_persistent_kernel()
    s.position_ = 0
    s.decode(3)
    s.close()
