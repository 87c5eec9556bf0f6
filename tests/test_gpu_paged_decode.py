"""A decode step of many sequences over the page pool (attention with head norm, RoPE and the cache write in one kernel), at the
edges of its ranges: one key, ranges that some warps or CTAs have no key of, pages of one and of odd sizes, every number of q
heads per kv head, both head dims, two to eight CTAs per row (one: test_gpu_paged_kernel.py), and contexts that the general kernels take.
A step at position n has to give what a prompt of n + 1 tokens gives, which other kernels compute."""
import numpy as np
import pytest

from buddy_mlir_b200 import ModelConfig, synthetic

pytestmark = pytest.mark.gpu
LENGTHS = [1, 2, 31, 32, 33, 64, 95, 127, 128, 257, 511]


@pytest.mark.parametrize("q_heads,kv_heads,D,qk_norm,page", [(12, 2, 128, False, 16), (8, 8, 64, False, 7), (4, 2, 128, True, 1), (6, 2, 64, True, 24),
                                                             (8, 2, 64, False, 16), (16, 2, 128, True, 33), (8, 1, 64, False, 5)])
def test_a_step_is_one_more_row_of_the_prompt(q_heads, kv_heads, D, qk_norm, page):
    from buddy_mlir_b200.session import BatchSession, ModelSession
    cfg = ModelConfig("paged", 256, 2, q_heads, kv_heads, D, 320, 400, 640, qkv_bias=not qk_norm, qk_norm=qk_norm)
    _, views = synthetic.make_f32_blob(cfg, 5)
    s = ModelSession(cfg)
    s.load_tensors(views, quantize_to="w8")
    rng = np.random.default_rng(q_heads + page)
    prompts = [rng.integers(0, cfg.vocab, n + 2) for n in LENGTHS]
    batch = BatchSession(s, 64, page, 2 * len(LENGTHS) * (640 // page + 1), 640)
    seqs = [batch.add() for _ in prompts]
    for q, p in zip(seqs, prompts):
        batch.prefill(q, p[:-2], want_logits=False)
    order = rng.permutation(len(seqs))
    whole = batch.add()
    for at in (-2, -1):             # two steps: the second reads the rows that the first wrote
        groups = (order, ) if at == -2 else (order[:1], order[1:4], order[4:])
        for group in groups:
            logits, _ = batch.decode([seqs[i] for i in group], [prompts[i][at] for i in group])
            for i, got in zip(group, logits):
                batch.remove(whole)
                whole = batch.add()
                end = len(prompts[i]) + at + 1
                want, _ = batch.prefill(whole, prompts[i][:end])
                # f32 sums of up to 512 keys in another order, approximate exponentials (2^-21) and three-digit GEMMs, two layers
                assert np.abs(got - want).max() / np.abs(want).max() < 2e-5, (LENGTHS[i], at)
    batch.close()
    s.close()


def test_contexts_beyond_the_kernels_ranges():
    from buddy_mlir_b200.session import BatchSession, ModelSession
    cfg = ModelConfig("long", 256, 1, 2, 1, 64, 320, 400, 9000)
    _, views = synthetic.make_f32_blob(cfg, 6)
    s = ModelSession(cfg)
    s.load_tensors(views, quantize_to="w8")
    rng = np.random.default_rng(9)
    batch = BatchSession(s, 3, 64, 3 * 141, 9000)
    for n in (8190, 8191, 8192):    # 8 x 1024 keys and one more
        tokens = rng.integers(0, cfg.vocab, n + 1)
        a, b = batch.add(), batch.add()
        batch.prefill(a, tokens[:-1], want_logits=False)
        got, _ = batch.decode([a], tokens[-1:])
        want, _ = batch.prefill(b, tokens)
        assert np.abs(got[0] - want).max() / np.abs(want).max() < 4e-5
        batch.remove(a)
        batch.remove(b)
    batch.close()
    s.close()
