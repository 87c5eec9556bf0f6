"""Orders inside kernels that keep a pass from waiting for itself, read off the CUDA sources (what goes wrong without them is a
wait on the GPU that never ends, so it is not tried there), and one pass on the GPU in which the kernels concerned meet."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import fake_runtime

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "buddy_mlir_b200", "csrc")


def kernels():
    """{name: body} of every __global__ function, comments removed."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, f)).read(), flags=re.S)
        for m in re.finditer(r"__global__\b[^;{]*?(\w+_kernel)\s*\([^{;]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            out[m.group(1)] = text[m.end():i]
    return out


def test_tensor_memory_is_allocated_before_the_next_kernel_may_start():
    users = {n: b for n, b in kernels().items() if "tcgen05.alloc" in b}
    assert set(users) >= {"gemm_i8_kernel", "prefill_attn_kernel"}
    for name, body in users.items():
        alloc, go = body.index("tcgen05.alloc"), body.find("kernel_go()")
        assert go < 0 or go > body.index("__syncthreads()", alloc), name


def test_weight_loads_of_a_public_call_stay_behind_the_callers_stream(tmp_path):
    """The GEMM loads weights before it waits: the kernel before it lets it start only after its own wait, unless the call is
    part of a session's pass."""
    start = re.search(r"void chain_start\(int in_pass\) \{(.*?)\n\}", open(os.path.join(CSRC, "gemm_tc.cu")).read(), re.S).group(1)
    assert re.sub(r"\s+", " ", start).strip() == "if (in_pass) kernel_go(); kernel_wait(); if (!in_pass) kernel_go();"
    bodies = kernels()
    for name in ("planes_kernel", "absmax_kernel"):
        assert bodies[name].split(";")[0].strip() == "chain_start(in_pass)" and "kernel_go" not in bodies[name]
    fake_runtime.run(tmp_path, "test_kernel_order", "first_kernels")


def first_kernels(fake):
    """What the host tells the first kernel of a call, over the stand-in runtime: (kernel, in_pass)."""
    from buddy_mlir_b200 import TINY_MEGA, _lib, synthetic
    from buddy_mlir_b200.session import ModelSession
    lib, seen = _lib.load(), []

    def launch(name, grid, args):
        for kernel, at in (("planes_kernel", 12), ("absmax_kernel", 8)):
            if kernel in name:
                seen.append((kernel, C.cast(args[at], C.POINTER(C.c_int))[0]))
    fake.on_launch(launch)
    buf = np.zeros(1 << 22, dtype=np.uint8)
    at = (buf.ctypes.data + 255) // 256 * 256
    w = _lib.Weight(_lib.W_I8, 0, 128, 64, at, at, _lib.F32, 0, None)
    _lib.check(lib.b200_gemm_w8(C.byref(w), at, 4, 128, at, 64, None, 0, None, 0.0, 0, at, 1 << 40, None))
    _lib.check(lib.b200_gemm_w8a8(C.byref(w), at, 4, 128, at, 64, at, 1 << 40, None))
    assert seen == [("planes_kernel", 0), ("absmax_kernel", 0)], seen
    for int8 in (0, 1):
        _, views = synthetic.make_f32_blob(TINY_MEGA, 3)
        s = ModelSession(TINY_MEGA)
        s.load_tensors(views, quantize_to="w8")
        s.set_activation_int8(bool(int8))
        del seen[:]
        s.prefill_rows(np.arange(5), 0, all_rows=False)
        assert seen and set(seen) == {("absmax_kernel" if int8 else "planes_kernel", 1)}
        s.close()


@pytest.mark.gpu
def test_weights_packed_just_before_the_call():
    import torch
    from buddy_mlir_b200 import _lib
    from gpu_util import dev, ptr, stream
    lib = _lib.load()
    rng = np.random.default_rng(2)
    M, N, K = 40, 512, 1024
    A = dev(rng.standard_normal((M, K)).astype(np.float32))
    q = [dev(rng.integers(-127, 128, (K, N)).astype(np.int8)) for _ in range(4)]
    one, packed = torch.ones(N, device="cuda"), torch.zeros(N * K, dtype=torch.uint8, device="cuda")
    w = _lib.Weight(_lib.W_I8, 0, K, N, packed.data_ptr(), one.data_ptr(), _lib.F32, 0, None)
    nb = lib.b200_gemm_w8_workspace_bytes(M, K)
    ws, out = torch.zeros(nb, dtype=torch.uint8, device="cuda"), torch.zeros(40, M, N, device="cuda")
    for i in range(40):
        _lib.check(lib.b200_pack_weight(_lib.W_I8, ptr(q[i % 4]), K, N, 1, ptr(packed), stream()))
        _lib.check(lib.b200_gemm_w8(C.byref(w), ptr(A), M, K, out[i].data_ptr(), N, None, 0, None, 0.0, 0, ptr(ws), nb, stream()))
    torch.cuda.synchronize()
    for i in range(40):
        want = A.double() @ q[i % 4].double()
        assert float((out[i].double() - want).abs().max() / want.abs().max()) < 4e-6


@pytest.mark.gpu
def test_head_dim_64_prefill_where_attention_and_gemm_fit_one_sm():
    import oracle_lib as orc
    from buddy_mlir_b200 import ModelConfig, synthetic
    from buddy_mlir_b200.session import ModelSession
    cfg = ModelConfig("hd64", 512, 4, 8, 2, 64, 1024, 900, 640)
    _, views = synthetic.make_f32_blob(cfg, 3)
    om = orc.OracleModel(cfg, views, kinds={n: "w8" for n in ("q", "k", "v", "o", "gate", "up", "down", "lm_head")})
    s = ModelSession(cfg)
    s.load_tensors(views, quantize_to="w8")
    tokens = np.random.default_rng(4).integers(0, cfg.vocab, 600)
    for _ in range(3):
        got = s.prefill_rows(tokens, 0, all_rows=False)
    for t in tokens:
        want = om.decode(int(t))
    # the tolerance stated for f32 logits of a row-batched pass over int8 weights
    assert np.abs(np.asarray(got).reshape(-1)[-cfg.vocab:] - want).max() / np.abs(want).max() < 1e-3
    s.close()
