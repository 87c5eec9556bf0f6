"""Orders inside kernels that keep a pass from waiting for itself, read off the CUDA sources (what goes wrong without them is a
wait on the GPU that never ends, so it is not tried there), and one pass on the GPU in which the kernels concerned meet."""
import os
import re

import numpy as np
import pytest

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
