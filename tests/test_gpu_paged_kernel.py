"""The batched decode attention by itself against f64, where the sessions' tests do not come: one CTA per row with many turns of its
warps, and ranges on both sides of what a CTA holds.  Called by its symbol, as are the kernels that it stands in for."""
import ctypes as C

import numpy as np
import pytest

from buddy_mlir_b200 import _lib

pytestmark = pytest.mark.gpu
i64, f32 = C.c_int64, C.c_float


class Step:
    """A decode step: rows of q|k|v without RoPE (frequencies of zero), their caches in shuffled pages."""

    def __init__(self, lens, q_heads, kv_heads, D, page, seed, scale=1.0, limit=0):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.lens, self.q, self.kv, self.D, self.page, self.M = lens, q_heads, kv_heads, D, page, len(lens)
        self.stride = (max(max(lens), limit) + page - 1) // page
        pages = [(n + page - 1) // page for n in lens]
        order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed)).to(torch.int32)
        self.table, at = torch.zeros(self.M, self.stride, dtype=torch.int32), 0
        for m, n in enumerate(pages):
            self.table[m, :n] = order[at:at + n]
            at += n
        self.table = self.table.cuda()
        self.k, self.v = (torch.randn(at, kv_heads, page, D, device="cuda", generator=g) for _ in range(2))
        self.ld = (q_heads + 2 * kv_heads) * D
        self.qkv = torch.randn(self.M, self.ld, device="cuda", generator=g)
        self.qkv[:, :q_heads * D] *= scale
        self.seq = torch.arange(self.M, dtype=torch.int32).cuda()
        self.pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32).cuda()
        self.freq = torch.zeros(D // 2, device="cuda")
        self.out = torch.zeros(self.M, q_heads * D, device="cuda")

    def takes(self):
        from gpu_util import ptr
        f = _lib.load()["_ZN4b20018paged_decode_takesEPKflS1_S1_iiiii"]
        f.restype = C.c_bool
        return f(ptr(self.qkv), i64(self.ld), ptr(self.k), ptr(self.v), self.q, self.kv, self.D, self.M, max(self.lens))

    def one_kernel(self):
        from gpu_util import ptr, stream
        _lib.check(_lib.load()["_ZN4b20019paged_decode_launchEPKflPfS2_S2_lS1_S1_S1_fiiiiPKiS4_S4_iiiP11CUstream_st"](
            ptr(self.qkv), i64(self.ld), ptr(self.k), ptr(self.v), ptr(self.out), i64(self.q * self.D), ptr(self.freq), None, None, f32(1e-6), self.q,
            self.kv, self.D, self.page, ptr(self.seq), ptr(self.pos), ptr(self.table), self.stride, self.M, max(self.lens), stream()))
        return self.out.clone()

    def three_kernels(self):
        import torch
        from gpu_util import ptr, stream
        lib, limit = _lib.load(), self.stride * self.page
        floats = lib["_ZN4b20024gqa_paged_scratch_floatsEiiii"]
        floats.restype = C.c_int64
        scratch = torch.zeros(floats(self.M, self.q, self.D, limit), device="cuda")
        _lib.check(lib["_ZN4b20020rope_kv_paged_launchEPflS0_S0_PKfS2_S2_fiiiiPKiS4_S4_iiP11CUstream_st"](
            ptr(self.qkv), i64(self.ld), ptr(self.k), ptr(self.v), ptr(self.freq), None, None, f32(1e-6), self.q, self.kv, self.D, self.page,
            ptr(self.seq), ptr(self.pos), ptr(self.table), self.stride, self.M, stream()))
        _lib.check(lib["_ZN4b20016gqa_paged_launchEPKflS1_S1_PfliiiiPKiS4_S4_iiS2_iiP11CUstream_st"](
            ptr(self.qkv), i64(self.ld), ptr(self.k), ptr(self.v), ptr(self.out), i64(self.q * self.D), self.q, self.kv, self.D, self.page, ptr(self.seq),
            ptr(self.pos), ptr(self.table), self.stride, self.M, ptr(scratch), self.M, limit, stream()))
        return self.out.clone()

    def exact(self):
        """In f64, after a step: the pools hold the newest rows."""
        import torch
        want = torch.empty(self.M, self.q * self.D, dtype=torch.float64, device="cuda")
        for m, n in enumerate(self.lens):
            at = self.table[m, :(n + self.page - 1) // self.page].long()
            k, v = (x[at].transpose(0, 1).reshape(self.kv, -1, self.D)[:, :n].double() for x in (self.k, self.v))
            q = self.qkv[m, :self.q * self.D].reshape(self.kv, -1, self.D).double()
            want[m] = (torch.softmax(q @ k.transpose(1, 2) / self.D ** 0.5, -1) @ v).reshape(-1)
        return want


def error(got, want):
    return float((got.double() - want).norm() / want.norm()), float(((got.double() - want).abs().amax(1) / want.abs().amax(1)).max())


def mixed(rng, rows, longest):
    return [longest] + [int(n) for n in rng.integers(1, longest + 1, rows - 1)]


# (rows, q heads, kv heads, D, longest): one CTA per row and kv head from 148 of them on, two from 74, eight up to 18; a CTA holds 1024 keys
@pytest.mark.parametrize("rows,q_heads,kv_heads,D,longest", [(19, 32, 8, 128, 1023), (19, 32, 8, 128, 1024), (80, 12, 2, 128, 700), (200, 12, 2, 128, 300),
                                                             (300, 8, 8, 64, 97), (74, 4, 2, 64, 1024), (37, 12, 2, 128, 2047), (10, 32, 8, 128, 2048),
                                                             (150, 8, 1, 128, 33), (160, 3, 1, 128, 259), (24, 12, 2, 128, 30),
                                                             (16, 4, 1, 64, 8191), (16, 4, 1, 64, 8192)])
def test_against_f64(rows, q_heads, kv_heads, D, longest):
    rng = np.random.default_rng(rows + longest)
    for scale in (1.0, 6.0):
        s = Step(mixed(rng, rows, longest), q_heads, kv_heads, D, 16, rows, scale)
        assert s.takes()
        got = s.one_kernel()
        norm, most = error(got, s.exact())
        others = error(s.three_kernels(), s.exact())[0]
        # f32 sums of D products and of up to 8192 weights, exponentials of 2 ulp of scores up to some 30 (rounded in powers of two)
        assert norm < 1e-6 and most < 2e-5
        # and no further off than the kernels that it stands in for, beyond what another order of the sums does
        assert norm < 1.15 * others, (norm, others)


def test_one_position_more_than_a_cta_holds():
    for rows, q_heads, kv_heads, longest in ((19, 32, 8, 1025), (10, 32, 8, 2049), (80, 12, 2, 1025), (16, 4, 1, 8193)):
        assert not Step([longest] + [5] * (rows - 1), q_heads, kv_heads, 128, 16, 1).takes()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 33, 34, 70, 129])
def test_infinite_values_stay_infinite(n, D):
    """An infinity in the newest value row, or in the last of a CTA's range: weights of zero are not multiplied by it."""
    s = Step([n, 257, n], 12, 2, D, 16, n, limit=300)
    s.qkv[0, (12 + 2) * D + 3] = float("inf")                                     # of the first row's kv head 0, dim 3
    for j in range(1, 257, 2):                                                     # every other old position of the second
        s.v[s.table[1, j // 16].long(), 1, j % 16, 5] = float("-inf")
    got = s.one_kernel().reshape(3, 12, D)
    assert (got[0, :6, 3] == float("inf")).all() and (got[1, 6:, 5] == float("-inf")).all()
    got[0, :6, 3] = got[1, 6:, 5] = 0
    assert got.isfinite().all()
