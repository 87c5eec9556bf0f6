"""The persistent decode kernel at the sizes where its plan can go wrong: fewer stream blocks than warps, ragged last
blocks and tiles, one key range and several, the new key first or last of a pass, each weight kind and a mix of them.
Reference: the CPU checker, step by step over a seeded cache prefix."""
import numpy as np
import pytest

import oracle_lib as orc
from buddy_mlir_b200 import TINY_MEGA, TINY_QWEN3, ModelConfig, synthetic
from buddy_mlir_b200.session import ModelSession

pytestmark = pytest.mark.gpu
LINEAR = ("q", "k", "v", "o", "gate", "up", "down", "lm_head")
# ragged everywhere: hidden 516 (no multiple of 128), ffn 1300, one q head per kv head, vocabulary of 16 k + 1
ODD = ModelConfig("odd", 516, 2, 3, 3, 128, 1300, 1601, 200)
# one kv head: the key ranges are spread over all CTAs
DEEP = ModelConfig("deep", 512, 2, 8, 1, 128, 1024, 2048, 2304)


def maxrel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("cfg,quant,group,positions", [
    (ODD, "w8", 0, (0, 1, 63, 64, 65, 199)), (TINY_MEGA, None, 0, (0, 62, 63, 64, 127, 128, 129)),
    (TINY_QWEN3, "w4", 128, (0, 31, 63, 64, 100)), (DEEP, "w8", 0, (5, 2047, 2048, 2303)), (DEEP, "w4", 128, (70, 2303))])
def test_steps_match_the_checker(cfg, quant, group, positions):
    _, views = synthetic.make_f32_blob(cfg, 7)
    kinds = {None: None, "w8": {n: "w8" for n in LINEAR}, "w4": {n: "w4g" for n in LINEAR}}[quant]
    om = orc.OracleModel(cfg, views, kinds=kinds)
    s = ModelSession(cfg)
    s.load_tensors(views, quantize_to=quant, group=group)
    assert s.uses_persistent_kernel()
    rng = np.random.default_rng(11)
    for b in range(2 * cfg.n_layers):
        pre = rng.standard_normal((cfg.kv_heads, cfg.max_len, cfg.head_dim)).astype(np.float32)
        om.kv[b][:] = pre
        s.kv_upload(b, pre, 0, cfg.max_len)
    for pos in positions:
        om.position = s.position_ = pos
        s.decode(17 + pos % 1000)
        want = om.decode(17 + pos % 1000)
        assert maxrel(s.logits_data(), want) < 1e-4, pos
        for b in range(2 * cfg.n_layers):
            assert maxrel(s.kv_download(b)[:, pos], om.kv[b][:, pos]) < 1e-4
    s.close()


def test_mixed_float_and_int8_projections():
    """The shipped w8a32 split: q, k, v f32, the rest int8."""
    cfg = TINY_MEGA
    _, views = synthetic.make_f32_blob(cfg, 5)
    floats, ints = synthetic.split_w8a32(cfg, views, lambda w: orc.quantize_per_channel(w, 8))
    om = orc.OracleModel(cfg, views, kinds={n: "w8" for n in synthetic.QUANTISED_BY_REFERENCE})
    s = ModelSession(cfg)
    s.load_blobs("w8a32", floats, ints)
    assert s.uses_persistent_kernel()
    for t in synthetic.prompt_tokens(cfg, 2, 5):
        s.decode(int(t))
        assert maxrel(s.logits_data(), om.decode(int(t))) < 1e-4
    s.close()


def test_steps_without_the_kernels_copy_of_the_weights():
    """A request that cannot be met takes the copy of the weights away and brings it back; the w8a8 arithmetic starts without it."""
    from buddy_mlir_b200 import _lib
    from buddy_mlir_b200.session import BatchSession
    cfg = TINY_MEGA
    _, views = synthetic.make_f32_blob(cfg, 5)
    floats, ints = synthetic.split_w8a32(cfg, views, lambda w: orc.quantize_per_channel(w, 8))
    om = orc.OracleModel(cfg, views, kinds={n: "w8" for n in synthetic.QUANTISED_BY_REFERENCE})
    s = ModelSession(cfg)
    s.load_blobs("w8a8", floats, ints)
    assert not s.uses_persistent_kernel()
    s.set_activation_int8(False)
    assert s.uses_persistent_kernel()
    for i, t in enumerate(synthetic.prompt_tokens(cfg, 2, 6)):
        if i == 2:
            with pytest.raises(_lib.B200Error):
                BatchSession(s, 1, 16, 1 << 24, 64)     # pools of 256 GB
            assert s.uses_persistent_kernel()
        s.decode(int(t))
        assert maxrel(s.logits_data(), om.decode(int(t))) < 1e-4
    s.close()
