"""The work whose speed matters to a user of this library: cases, inputs, one pass, and what a pass cannot do without.

Every case goes through a public entry point: the device-pointer C ABI (`b200_*`), the per-op external kernels on host
buffers (`_mlir_ciface_buddy_*`), the sessions (`ModelSession`, `BatchSession`) and the model entry that buddy-mlir's
generated host calls (`EntrySession`).  Shapes are those of the repository's own configurations
(DEEPSEEK_R1_1P5B, QWEN3_8B) and of its GEMV / GEMM sweeps.
"""
import ctypes as C
import math

import numpy as np
import torch

from buddy_mlir_b200 import DEEPSEEK_R1_1P5B, QWEN3_8B, _lib, memref, synthetic
from buddy_mlir_b200.model_entry import EntrySession
from buddy_mlir_b200.session import BatchSession, ModelSession

MODELS = {"1.5b": DEEPSEEK_R1_1P5B, "8b": QWEN3_8B}
DTYPES = {"f32": (torch.float32, _lib.F32), "f16": (torch.float16, _lib.F16), "bf16": (torch.bfloat16, _lib.BF16)}


def listed():
    return [
        # one decode projection of one layer (o of the 1.5B model), as a host that issues the step itself calls it:
        # nothing but latency
        {"name": "gemv_i8_o", "op": "gemv", "weights": "i8", "M": 1, "N": 1536, "K": 1536, "group": 0, "x": "f32", "calls": 1},
        # int4 group-128 FFN projection for a handful of rows (speculative tokens, a few users), one call per layer
        {"name": "gemv_u4_ffn", "op": "gemv", "weights": "u4", "M": 5, "N": 14336, "K": 4096, "group": 128, "x": "bf16", "calls": 8},
        # prefill: RMSNorm, gate and up of one layer, SiLU pair, at the reference's prompt length
        {"name": "gemm_gate_up", "op": "gemm", "M": 1024, "N": 17920, "K": 1536, "norm": True, "silu": True},
        # int8 activations (the reference's w8a8 graphs), down projection of a ragged prompt
        {"name": "gemm_w8a8_down", "op": "w8a8", "M": 333, "N": 1536, "K": 8960},
        # the same decode matmul as compiled buddy-mlir code calls it: host buffers behind MemRef descriptors
        {"name": "abi_gemv_gate", "op": "abi", "M": 1, "N": 8960, "K": 1536},
        # a chat step early in a conversation: one token in, logits on the host
        {"name": "decode_i8", "op": "decode", "model": "1.5b", "weights": "w8", "ctx": 97},
        # greedy generation at the end of a 1024-token context, tokens only
        {"name": "generate_i8_1k", "op": "generate", "model": "1.5b", "weights": "w8", "ctx": 1008, "steps": 16},
        # unquantised weights (the reference's default variant)
        {"name": "decode_f32", "op": "decode", "model": "1.5b", "weights": "f32", "ctx": 257},
        # the large model, int4 group-128, at the end of a 4096-token context
        {"name": "decode_u4_8b", "op": "decode", "model": "8b", "weights": "w4", "ctx": 4000},
        # a long prompt of ragged length, logits of its last row
        {"name": "prefill_1000", "op": "prefill", "model": "1.5b", "rows": 1000},
        # a serving round over the paged cache: two dozen prompts come in, all are decoded together
        {"name": "batch_serve", "op": "batch", "model": "1.5b", "seqs": 24, "shortest": 32, "longest": 700, "steps": 32},
        # buddy-mlir's generated host: the w8a32 entry, host cache and logits, eight tokens of a reply
        {"name": "entry_w8a32", "op": "entry", "model": "1.5b", "ctx": 301, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["gemv", "gemv", "gemm", "w8a8", "abi", "decode", "decode", "generate", "prefill", "batch", "entry"])
    if op == "gemv":
        kind = rng.choice(["i8", "u4"])
        k = _log(rng, 512, 14336)
        n = _log(rng, 500, 152000)
        k = k // 128 * 128 if kind == "u4" else k // 16 * 16
        m = rng.choice([1, 1, 1, rng.randint(2, 16)])
        return {"op": op, "weights": kind, "M": m, "N": n if kind == "i8" else n // 2 * 2, "K": k, "group": 128 if kind == "u4" else 0,
                "x": rng.choice(["f32", "f32", "f16", "bf16"]), "calls": max(1, min(8, int(4e8 / (n * k))))}
    if op in ("gemm", "w8a8"):
        m, k, n = _log(rng, 17, 2048), _log(rng, 512, 8960) // 64 * 64, _log(rng, 500, 20000)
        if op == "w8a8":
            return {"op": op, "M": m, "N": n, "K": k}
        return {"op": op, "M": m, "N": n // 8 * 8, "K": k, "norm": rng.random() < 0.5, "silu": rng.random() < 0.3}
    if op == "abi":
        return {"op": op, "M": rng.choice([1, 1, rng.randint(2, 16)]), "N": _log(rng, 500, 18000), "K": _log(rng, 512, 8960) // 16 * 16}
    if op == "decode":
        model, weights = rng.choice([("1.5b", "w8"), ("1.5b", "w8"), ("1.5b", "f32"), ("8b", "w4")])
        return {"op": op, "model": model, "weights": weights, "ctx": _log(rng, 8, MODELS[model].max_len - 1)}
    if op == "generate":
        steps = rng.randint(8, 32)
        return {"op": op, "model": "1.5b", "weights": "w8", "ctx": _log(rng, 8, 1024 - steps), "steps": steps}
    if op == "prefill":
        return {"op": op, "model": "1.5b", "rows": _log(rng, 16, 2048)}
    if op == "batch":
        longest = _log(rng, 64, 700)
        return {"op": op, "model": "1.5b", "seqs": rng.randint(2, 24), "shortest": rng.randint(16, longest), "longest": longest,
                "steps": rng.randint(8, 32)}
    return {"op": op, "model": "1.5b", "ctx": _log(rng, 8, 1000), "steps": rng.randint(4, 8)}


# ---- inputs ------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(gen, *shape, std=1.0):
    return torch.empty(*shape, device="cuda").normal_(0.0, std, generator=gen)


#: what a serving process keeps between requests: the weights of its model on the host (one model at a time), and the
#: session of a model whose calls carry their whole input with them (a prompt), shared by every request
_kept = {}


def _keep(key, make):
    if key not in _kept:
        for k in [k for k in _kept if k[0] == key[0]]:
            v = _kept.pop(k)
            if hasattr(v, "close"):
                v.close()
        _kept[key] = make()
    return _kept[key]


def _host_tensors(cfg):
    """{(name, layer): f32 array} as ModelSession.load_tensors takes it: N(0, 0.02) weights, norms around 1.  The
    tensors are windows of one page-locked pool (no checkpoint is at hand; the values only have to be distributed so)."""
    def make():
        longest = max(int(np.prod(s)) for _, _, s in synthetic.tensor_list(cfg))
        pool = torch.empty(longest + (1 << 22), dtype=torch.float32, pin_memory=True)
        pool.copy_(_randn(_gen(1), pool.numel(), std=0.02))
        flat, views = pool.numpy(), {"pool": pool}
        at = 0
        for name, layer, shape in synthetic.tensor_list(cfg):
            n = int(np.prod(shape))
            at = (at + 1009 * 64) % (flat.size - n)
            v = flat[at:at + n].reshape(shape)
            views[(name, layer)] = synthetic.inv_freq(cfg) if name == "inv_freq" else v + np.float32(1) if name.endswith("norm") else v
        return views
    return _keep(("tensors", cfg), make)


def _session(cfg, weights):
    s = ModelSession(cfg)
    s.load_tensors(_host_tensors(cfg), quantize_to=None if weights == "f32" else weights, group=128 if weights == "w4" else 0)
    return s


def _kv_rows(cfg, gen, n):
    """n rows of every cache buffer, [kv_heads, max_len, head_dim] on the host, one buffer after the other."""
    host = torch.zeros(cfg.kv_heads, cfg.max_len, cfg.head_dim, pin_memory=True)
    for _ in range(2 * cfg.n_layers):
        host[:, :n].copy_(_randn(gen, cfg.kv_heads, n, cfg.head_dim))
        yield host.numpy()


def _w8a32_blobs(cfg):
    """The two files of the w8a32 variant (arg0.data, arg1.data) in memory."""
    def make():
        gen, floats, scales, ints = _gen(1), [], [], []
        for name, _, shape in synthetic.tensor_list(cfg):
            if name in synthetic.QUANTISED_BY_REFERENCE:
                ints.append(_randn(gen, *shape, std=28.0).round_().clamp_(-127, 127).to(torch.int8).cpu().numpy().reshape(-1))
                scales.append(np.full(shape[1], 0.02 / 28, dtype=np.float32))
            elif name == "inv_freq":
                floats.append(synthetic.inv_freq(cfg))
            else:
                floats.append((_randn(gen, *shape, std=0.02) + (1.0 if name.endswith("norm") else 0.0)).cpu().numpy().reshape(-1))
        return np.concatenate(floats + scales), np.concatenate(ints)
    return _keep(("tensors", cfg, "w8a32"), make)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _packed_i8(lib, gen, K, N):
    """Weights N(0, 0.02), quantised per channel and packed by the library."""
    W = _randn(gen, K, N, std=0.02)
    q = torch.empty(K, N, dtype=torch.int8, device="cuda")
    scale = torch.empty(N, device="cuda")
    packed = torch.zeros(lib.b200_packed_row_bytes(_lib.W_I8, K) * N, dtype=torch.uint8, device="cuda")
    _lib.check(lib.b200_quantize_per_channel(W.data_ptr(), K, N, 8, q.data_ptr(), scale.data_ptr(), _stream()))
    _lib.check(lib.b200_pack_weight(_lib.W_I8, q.data_ptr(), K, N, 1, packed.data_ptr(), _stream()))
    return packed, scale


def _packed_u4(lib, gen, K, N, G):
    W = _randn(gen, K, N, std=0.02)
    codes = torch.empty(K, N // 2, dtype=torch.uint8, device="cuda")
    raw = torch.empty(K // G, N, dtype=torch.float16, device="cuda")
    scale = torch.empty(N, K // G, dtype=torch.float16, device="cuda")
    packed = torch.zeros(lib.b200_packed_row_bytes(_lib.W_U4, K) * N, dtype=torch.uint8, device="cuda")
    _lib.check(lib.b200_quantize_w4_group(W.data_ptr(), K, N, G, codes.data_ptr(), raw.data_ptr(), _stream()))
    _lib.check(lib.b200_pack_weight(_lib.W_U4, codes.data_ptr(), K, N, 0, packed.data_ptr(), _stream()))
    _lib.check(lib.b200_pack_scales(raw.data_ptr(), _lib.F16, K // G, N, scale.data_ptr(), _stream()))
    return packed, scale


def prepare(case, seed):
    lib, gen, op = _lib.load(), _gen(seed), case["op"]
    s = dict(case, lib=lib)
    if op in ("gemv", "gemm", "w8a8", "abi"):
        M, N, K = case["M"], case["N"], case["K"]
    if op == "gemv":
        dt, code = DTYPES[case["x"]]
        s["x"] = _randn(gen, M, K).to(dt)
        s["weights"], s["y"], s["calls"] = [], [], []
        for _ in range(case["calls"]):
            kind = _lib.W_I8 if case["weights"] == "i8" else _lib.W_U4
            w, scale = _packed_i8(lib, gen, K, N) if kind == _lib.W_I8 else _packed_u4(lib, gen, K, N, case["group"])
            y = torch.empty(M, N, device="cuda")
            s["weights"].append((w, scale))
            s["y"].append(y)
            s["calls"].append((_lib.Weight(kind, case["group"], K, N, w.data_ptr(), scale.data_ptr(),
                                           _lib.F32 if kind == _lib.W_I8 else _lib.F16, 0, None),
                               _lib.GemvArgs(s["x"].data_ptr(), code, _lib.F32, K, N, y.data_ptr(), None, None, 0.0, M, 0, 0)))
    elif op in ("gemm", "w8a8"):
        s["A"] = _randn(gen, M, K)
        s["packed"] = _packed_i8(lib, gen, K, N)
        s["w"] = _lib.Weight(_lib.W_I8, 0, K, N, s["packed"][0].data_ptr(), s["packed"][1].data_ptr(), _lib.F32, 0, None)
        s["ld"] = N // 2 if case.get("silu") else N
        s["C"] = torch.empty(M, s["ld"], device="cuda")
        s["norm"] = 1.0 + _randn(gen, K, std=0.02) if case.get("norm") else None
        s["bytes"] = lib.b200_gemm_w8_workspace_bytes(M, K) if op == "gemm" else lib.b200_gemm_w8a8_workspace_bytes(M, K)
        s["workspace"] = torch.zeros(s["bytes"], dtype=torch.uint8, device="cuda")
    elif op == "abi":
        s["A"] = _randn(gen, M, K).cpu().numpy()
        s["W"] = _randn(gen, K, N, std=28.0).round_().clamp_(-127, 127).to(torch.int8).cpu().numpy()
        s["scale"] = np.full((1, N), 0.02 / 28, dtype=np.float32)
        memref.buddy_gemv_w8_f32(s["A"], s["W"], s["scale"])        # the library keeps its device copy of a weight
    else:
        cfg = MODELS[case["model"]]
        ids = np.random.default_rng(seed)
        if op in ("decode", "generate"):
            s["session"] = _session(cfg, case["weights"])
            for b, rows in enumerate(_kv_rows(cfg, gen, case["ctx"])):
                s["session"].kv_upload(b, rows, 0, case["ctx"])
            s["token"] = int(ids.integers(cfg.vocab))
        elif op == "prefill":
            cfg = cfg.with_(max_len=2048)
            s["session"] = _keep(("prompts", cfg), lambda: _session(cfg, "w8"))
            s["tokens"] = ids.integers(0, cfg.vocab, case["rows"]).astype(np.int32)
        elif op == "batch":
            cfg = cfg.with_(max_len=2048)
            model = _keep(("prompts", cfg), lambda: _session(cfg, "w8"))
            pages = case["seqs"] * ((case["longest"] + case["steps"] + 15) // 16)
            s["batch"] = BatchSession(model, case["seqs"], 16, pages, case["longest"] + case["steps"])
            s["prompts"] = [ids.integers(0, cfg.vocab, int(n)).astype(np.int32)
                            for n in ids.integers(case["shortest"], case["longest"] + 1, case["seqs"])]
            s["tokens"] = ids.integers(0, cfg.vocab, (case["steps"], case["seqs"])).astype(np.int32)
        else:
            s["session"] = EntrySession(cfg, "w8a32", _w8a32_blobs(cfg))
            for b, rows in enumerate(_kv_rows(cfg, gen, case["ctx"])):
                np.copyto(s["session"].kv[b][0], rows)
            s["tokens"] = ids.integers(0, cfg.vocab, case["steps"])
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(s):
    lib, op = s["lib"], s["op"]
    if op == "gemv":
        for w, a in s["calls"]:
            _lib.check(lib.b200_gemv(C.byref(w), C.byref(a), _stream()))
        return s["y"]
    if op == "gemm":
        _lib.check(lib.b200_gemm_w8(C.byref(s["w"]), s["A"].data_ptr(), s["M"], s["K"], s["C"].data_ptr(), s["ld"], None, 0,
                                    s["norm"].data_ptr() if s["norm"] is not None else None, 1e-6, int(s["silu"]),
                                    s["workspace"].data_ptr(), s["bytes"], _stream()))
        return s["C"]
    if op == "w8a8":
        _lib.check(lib.b200_gemm_w8a8(C.byref(s["w"]), s["A"].data_ptr(), s["M"], s["K"], s["C"].data_ptr(), s["ld"],
                                      s["workspace"].data_ptr(), s["bytes"], _stream()))
        return s["C"]
    if op == "abi":
        return memref.buddy_gemv_w8_f32(s["A"], s["W"], s["scale"])
    if op == "decode":
        session = s["session"]
        session.position_ = s["ctx"]                 # the same step again: it writes cache row ctx and reads rows 0..ctx
        session.decode(s["token"])
        return session.logits_data()
    if op == "generate":
        s["session"].position_ = s["ctx"]
        return s["session"].generate(s["token"], s["steps"])
    if op == "prefill":
        return s["session"].prefill_rows(s["tokens"], 0, all_rows=False)
    if op == "batch":
        batch = s["batch"]
        seqs = [batch.add() for _ in s["prompts"]]
        first = [batch.prefill(q, p, want_logits=False)[1] for q, p in zip(seqs, s["prompts"])]
        ids = [batch.decode(seqs, t, want_logits=False)[1] for t in s["tokens"][:-1]]   # tokens of given continuations
        logits, last = batch.decode(seqs, s["tokens"][-1])
        for q in seqs:
            batch.remove(q)
        return {"ids": np.concatenate([np.asarray(first, dtype=np.int32)] + ids + [last]), "logits": logits}
    session, logits = s["session"], []
    session.position_ = s["ctx"]
    for t in s["tokens"]:
        session.decode(int(t))
        logits.append(session.logits.copy())
    rows = np.stack([k[0, :, s["ctx"]:s["ctx"] + s["steps"]] for k in session.kv])      # the cache rows of the reply
    return {"logits": np.stack(logits), "kv": rows}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _linear_elements(cfg):
    """Elements of the linear layers of all layers, and of the lm_head."""
    per = cfg.hidden * (cfg.q_dim + 2 * cfg.kv_dim) + cfg.q_dim * cfg.hidden + 3 * cfg.hidden * cfg.ffn
    return cfg.n_layers * per, cfg.hidden * cfg.vocab


def _weight_bytes(cfg, weights):
    lin, head = _linear_elements(cfg)
    if weights == "w8a32":
        qkv = cfg.n_layers * cfg.hidden * (cfg.q_dim + 2 * cfg.kv_dim)
        return 4 * qkv + (lin - qkv) + head
    return (lin + head) * {"f32": 4.0, "w8": 1.0, "w4": 0.5 + 2 / 128}[weights]


def _attention(cfg, rows):
    """(bytes, flops) of attention for one query row against `rows` cache rows, all layers."""
    return cfg.n_layers * 2 * cfg.kv_dim * 4 * rows, cfg.n_layers * 4 * cfg.q_dim * rows


def work(case):
    op = case["op"]
    if op == "gemv":
        M, N, K, n = case["M"], case["N"], case["K"], case["calls"]
        w = N * K + 4 * N if case["weights"] == "i8" else N * K // 2 + 2 * N * (K // case["group"])
        return {"bytes": n * (w + M * K * (4 if case["x"] == "f32" else 2) + 4 * M * N), "flops": n * 2 * M * N * K}
    if op in ("gemm", "w8a8"):
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": N * K + 4 * N + 4 * M * K + 4 * M * (N // 2 if case.get("silu") else N), "flops": 2 * M * N * K}
    if op == "abi":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": N * K + 4 * N + 4 * M * (K + N), "flops": 2 * M * N * K}
    cfg = MODELS[case["model"]]
    lin, head = _linear_elements(cfg)
    if op in ("decode", "generate", "entry"):
        b = f = 0
        for i in range(case.get("steps", 1)):
            kb, kf = _attention(cfg, case["ctx"] + i + 1)
            b += _weight_bytes(cfg, case.get("weights", "w8a32")) + kb + 4 * cfg.vocab
            f += 2 * (lin + head) + kf
        return {"bytes": b, "flops": f}
    if op == "prefill":
        n = case["rows"]
        kb, _ = _attention(cfg, n)
        _, kf = _attention(cfg, n * (n + 1) // 2)
        return {"bytes": lin + head + 2 * kb + 4 * n * cfg.hidden, "flops": 2 * (n * lin + head) + kf}
    n, mean = case["seqs"], (case["shortest"] + case["longest"]) / 2
    kb, kf = _attention(cfg, mean + case["steps"] / 2)
    _, pf = _attention(cfg, mean * (mean + 1) / 2)
    return {"bytes": (case["steps"] + 1) * (lin + head) + n * case["steps"] * kb,
            "flops": n * (2 * (mean * lin + head) + pf) + n * case["steps"] * (2 * (lin + head) + kf)}


def tolerance(case):
    op = case["op"]
    if op == "w8a8":
        return "exact"               # integer sums, one rounding per element: bit-identical by contract
    if op in ("gemv", "abi"):
        return {"rel": 1e-5}         # f32 sums in another order
    if op == "gemm":
        return {"rel": 2e-5}         # f32 activations as two bf16 terms (2^-17 each), f32 sums
    if op == "generate":
        return {"rel": 0.0, "differ": 0.0}
    if op in ("decode", "entry"):
        return {"rel": 1e-4}         # f32 sums through 28 or 36 layers
    return {"rel": 2e-4, "differ": 0.01}     # the two-term GEMM through 28 layers; ids of near-equal logits may flip
