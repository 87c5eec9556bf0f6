"""The prefill attention on the tensor cores at the sizes where its plan can go wrong: row tiles that end inside a query row
(group sizes 1, 3, 6), ragged last tiles of rows and keys, one key range per row tile and several, histories that end at a
tile's edge, both head sizes, pages.  Reference: the CPU checker, row by row over a seeded cache prefix."""
import numpy as np
import pytest

import oracle_lib as orc
from buddy_mlir_b200 import ModelConfig, synthetic
from buddy_mlir_b200.session import BatchSession, ModelSession

pytestmark = pytest.mark.gpu


def maxrel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("G,kvh,D,pos0,rows", [
    (1, 2, 64, 0, 64), (6, 2, 128, 0, 127), (6, 1, 128, 450, 65), (3, 2, 64, 63, 129), (4, 1, 128, 700, 68), (8, 2, 64, 128, 64),
    (2, 3, 128, 1, 200)])
def test_rows_match_the_checker(G, kvh, D, pos0, rows):
    cfg = ModelConfig("attn", 256, 1, G * kvh, kvh, D, 320, 500, 768)
    _, views = synthetic.make_f32_blob(cfg, 3)
    om = orc.OracleModel(cfg, views)
    s = ModelSession(cfg)
    s.load_tensors(views)
    rng = np.random.default_rng(4)
    for b in range(2):
        pre = (2 * rng.standard_normal((kvh, cfg.max_len, D))).astype(np.float32)
        om.kv[b][:] = pre
        s.kv_upload(b, pre, 0, cfg.max_len)
    tokens = rng.integers(0, cfg.vocab, rows)
    got = s.prefill_rows(tokens, pos0)
    om.position = pos0
    for i, t in enumerate(tokens):
        assert maxrel(got[i], om.decode(int(t))) < 1e-4, i
    s.close()


@pytest.mark.parametrize("page,chunks", [(7, (65, 64)), (16, (64, 190, 66))])
def test_pages_match_the_checker(page, chunks):
    cfg = ModelConfig("attn", 256, 1, 6, 1, 128, 320, 500, 400)
    _, views = synthetic.make_f32_blob(cfg, 3)
    om = orc.OracleModel(cfg, views)
    s = ModelSession(cfg)
    s.load_tensors(views)
    bs = BatchSession(s, max_seqs=2, page_size=page, n_pages=80, max_context=cfg.max_len)
    seq, rng = bs.add(), np.random.default_rng(4)
    for n in chunks:
        tokens = rng.integers(0, cfg.vocab, n)
        got, _ = bs.prefill(seq, tokens)
        for t in tokens:
            want = om.decode(int(t))
        assert maxrel(got, want) < 1e-4
    bs.close()
    s.close()
