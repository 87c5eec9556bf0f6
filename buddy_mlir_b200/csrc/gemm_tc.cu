// Dense weight-only-quantised GEMM on the 5th-generation tensor cores:
//   C[M,N] = A[M,K] (f32) * dequant(W)[N,K]^T, per-channel scale in the epilogue.
//
// This is the prefill / batched-decode path.  buddy-mlir's prefill GEMM
// (midend/lib/Conversion/MatMulOptimization/MatMulBlisVectorization.cpp:367-530)
// dequantises w = float(q) * scale while it packs B and then runs f32 FMAs; here
// the integer part and the scale are separated (sum_k a*q, then * scale[n]),
// which is the same product up to f32 rounding (the parity tests hold it to
// 1e-3 of the CPU restatement, as for the decode path).
//
// Operands.  Both are int8 and go from memory to the tensor cores as they are stored (tcgen05.mma kind::i8, s32
// accumulators in tensor memory).  The weights are the packed decode rows.  A row of activations is a 24-bit fixed-point
// number per element, in units of a power of two taken from the row's largest magnitude, and its three base-256 digits are
// three neighbouring rows of the digit operand, in the k order of the packed weights.  All products and sums are exact
// integers; the epilogue adds the digits' sums in f32.
// Two bf16 terms per activation and weights converted to bf16, the form before this one, kept 2^-17 of each element; three
// digits keep 2^-23 of the row's largest, which is less where a few channels of a row are far above the rest.  Such rows are
// wide: six digits, in passes of their own over the tile (planes_kernel says which rows).
// Relative error (2-norm, against f64) of the columns that do not use a channel R times the rest, 256 x 1536 x 1536:
//   R            1        30       100      1000     10000
//   now          1.7e-7   1.1e-6   9.4e-7   4.0e-7   8.1e-8
//   three digits 3.2e-7   3.2e-6   1.0e-5   1.1e-4   9.9e-4    (for every row, 23 bits)
//   two bf16     2.5e-6 for all; f32 products and sums 7.0e-7
// Time with no wide row / one / all, us, weights from memory: 1024 x 17920 x 1536 69 / 85 / 180, 1000 x 1536 x 8960 40 / 65 / 109,
// 24 x 17920 x 1536 12.6 / 19 / 22.
//
// W8A8 (b200_gemm_w8a8) is the same kernel with one digit per activation.
//
// Tiles.  The weights are the operand with M rows (lanes of tensor memory), the digits the one with N columns: a thread of the
// epilogue then holds one channel, with all digits of an activation in neighbouring registers, so it adds them, scales and
// stores without shared memory, a warp 128 bytes of an output row at a time; gate and up are neighbouring lanes.  (Digits as M
// rows: the sums of a row lie in three lanes and go through 66 KB of shared memory.)  The two CTAs of a pair (cta_group::2) work
// on 256 channels x up to 84 activation rows: each brings its 128 weight rows and half of the digit rows, 32 KB per 128 k, which
// at 64 bytes per clock takes as long as the products (512 clocks); a CTA by itself brings 48 KB for as many products.
// The kernel stays on its SMs for all tiles: warp 0 loads (TMA, no multicast), warp 1 issues tcgen05.mma, sixteen warps are the
// epilogue of one accumulator while the products of the next tile go to the other.  What an epilogue needs from memory it asks
// for a tile ahead: with loads in its loop over the rows a tile took 16600 clocks, not 6100 (L2 answers late under these loads).
// Bound by the operands' way out of L2: a launch of 1000 x 17920 x 1536 brings 674 MB to the SMs, 46 bytes a clock and SM (10 TB/s;
// make_plan counts 45), while the tensor pipe is active in 71 % of the cycles and L2's slices in 41 %; and by the clock, which
// falls to 1.7 GHz.  1024 x 17920 x 1536 69 us with the digits' own pass, 108 us as CTAs of 128 x 256 for a tile each; 2.9 POP/s of the
// padded tiles.  1000 x 1536 x 8960: 40 us (49), 366 x 17920 x 1536: 31 us (50), W8A8 2048 x 8960 x 8960: 143 us (213).
// Few tiles: the k range is cut over the pairs of a cluster, whose sums meet in shared memory: make_plan().  The weight loads
// start before the activations are there (programmatic dependent launch behind the kernel that makes the digits; chain_start says
// what keeps them behind the caller's earlier work).
//
// Every wait is bounded (poll count and wall time); on expiry the CTA records
// an error, all roles fall through, tensor memory is released and the host
// call fails.
#include "common.cuh"
#include "gemv_mma.cuh"
#include "tensor_core.cuh"

#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <mutex>

namespace b200 {

namespace {

constexpr int BM = 128;                        // channels of a CTA's tile
constexpr int BK = 128;                        // int8 per k block: one 128-byte swizzle row
constexpr int kPlanes = 3, kWidePlanes = 6;    // digits per activation; of rows that need more
constexpr int kMaxStages = 8;
constexpr int kSms = 148, kPairs = kSms / 2;
constexpr int kMaxSplits = 4;                  // along k: clusters of up to eight CTAs
constexpr int kHeadBytes = 256;                // workspace head: error word, scales of W8A8
constexpr int kHeadWords = 1;                  // of it, cleared at the start of a call: the error word
constexpr uint32_t kWBytes = BM * BK;

struct Bars {
  uint64_t full[kMaxStages];   // TMA bytes of the stage have landed (in both CTAs of a pair: the first one's)
  uint64_t empty[kMaxStages];  // the tensor core is done with the stage
  uint64_t acc_full[2];        // an accumulator's MMAs have completed
  uint64_t acc_empty[2];       // the epilogue warps (of both CTAs) have read it
  uint64_t sums;               // split k: the sums of all shares for this CTA's rows are here
  uint32_t tmem_base;
  int abort_flag;
};

// (of a pair: the barrier may be the other CTA's)
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap *map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
// kind::i8 instruction descriptor: D = s32, A = B = s8, both K-major, M = 2 x 128 channels, N = nc digits.
__device__ __forceinline__ uint32_t mma_desc(int nc) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nc >> 3) << 17) | ((uint32_t)(2 * BM >> 4) << 24);
}
// Executed by a whole warp in uniform control flow (the operands then live in uniform registers), issued by the lane whose
// `leader` is set.
__device__ __forceinline__ void mma_i8(uint32_t leader, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, l;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 l, %5, 0;\n"
      " @l tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {   // the same shared-memory place in a CTA of the cluster
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Arrives at `bar` in both CTAs of the pair when the MMAs issued so far have completed.
__device__ __forceinline__ void commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)(3u << (cluster_rank() & ~1u)))
               : "memory");
}
__device__ __forceinline__ void sync_cluster() {   // all its threads
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Eight columns of this warp's 32 lanes of tensor memory
__device__ __forceinline__ void tmem_load(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr)
               : "memory");
}
struct GemmParams {
  int M, N, K;                 // K: multiple of 64
  const float *scale, *bias;   // [N], bias may be null
  const float *row_scale;      // digits: [M], negative for wide rows; W8A8: one value
  const float *residual;       // [M, ldr] or null; may alias C
  float *C;                    // [M, ldc]
  int64_t ldc, ldr;
  int silu_pairs;              // columns (2j, 2j+1) are (gate_j, up_j): C[m, j] = silu(g) * u, ldc counts N/2 columns
  int splits;                  // CTAs (pairs) along K per tile: those of a cluster, which then has one tile
  int share_rows;              // rows that each of them completes
  int tiles, m_tiles;          // the row tiles of a column tile are neighbours
  int stages;
  int *error;
  int nc, rows;                // digits (columns) and activation rows of a tile
  int cols;                    // of tensor memory: a power of two, two accumulators
};

struct Tile {
  int n0, m0, rows;
};
__device__ __forceinline__ Tile tile_at(const GemmParams &p, int w) {
  const int nt = w / p.m_tiles, m0 = (w - nt * p.m_tiles) * p.rows;
  return {nt * (2 * BM), m0, min(p.rows, p.M - m0)};
}
// The row scales of a tile (lane l: rows l, l + 32, l + 64; a row that is not there: 0), requested a tile ahead of their use.
struct RowScales {
  float v[3];
  __device__ __forceinline__ void load(const GemmParams &p, int m0, int rows) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      v[j] = 32 * j + lane < rows ? __ldcg(p.row_scale + m0 + 32 * j + lane) : 0.f;
  }
  // Which halves of the rows have wide rows: those halves are passes of their own.
  __device__ __forceinline__ uint32_t wide_halves(const GemmParams &p) const {
    const int lane = threadIdx.x & 31, half = (p.rows + 1) >> 1;
    uint32_t h = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (signbit(v[j]))
        h |= 32 * j + lane < half ? 1u : 2u;
    return __reduce_or_sync(0xffffffffu, h);
  }
  __device__ __forceinline__ float at(int r0) const { return r0 < 32 ? v[0] : r0 < 64 ? v[1] : v[2]; }   // rows r0 & ~31 ..
};

// silu(g) * u.  The operations, their order and roundings are the reference's (subgraph0_decode_simplify.mlir:226-231: (g * sigmoid(g)) *
// u) and those of b200_silu_mul.  d = 1 + e^-g; __frcp_rn is 1 / d rounded to nearest.
__device__ __forceinline__ float silu_of(float g, float u, float d) { return __fmul_rn(__fmul_rn(g, __frcp_rn(d)), u); }

// ---- epilogue ----------------------------------------------------------------------------------------------------------------
enum { kEither, kSilu, kPlain };   // STORE: SiLU pairs, which have no residual, or not; kEither: p.silu_pairs says
// A warp reads the 32 lanes of tensor memory that match its rank within its warpgroup, a lane one channel; the warps that share a
// lane quarter take CR rows of the tile in turn.
constexpr int CR = 8;
constexpr int kEpiWarps = 16, kGroups = kEpiWarps / 4, kThreads = 64 + 32 * kEpiWarps;
struct Channel {
  int n;               // this lane's
  bool in;
  float scale, bias;
  __device__ __forceinline__ Channel(const GemmParams &p, int channel) : n(channel), in(channel < p.N) {
    scale = __ldg(p.scale + min(n, p.N - 1));
    bias = p.bias ? __ldg(p.bias + min(n, p.N - 1)) : 0.f;
  }
};
// Sums of N rows from row m of C on -> results.  rs: row scales, that of row i in lane `from` + i (W8A8: the one scale).  ALL: all
// N rows are stored, otherwise those whose bit of `live` is set.
template <bool PLANES, int STORE, bool ALL, int N>
__device__ __forceinline__ void finish_rows(const GemmParams &p, const Channel &c, int m, float (&y)[N], float rs, int from, uint32_t live,
                                            const float (&res)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (PLANES)
      y[i] = __fmul_rn(__fmul_rn(y[i], fabsf(__shfl_sync(0xffffffffu, rs, from + i))), c.scale);
    else   // linalg.py:12836-12846: float(acc) * (act_scale * weight_scale[n])
      y[i] = __fmul_rn(__int2float_rn(__float_as_int(y[i])), __fmul_rn(rs, c.scale));
  }
  if (p.bias) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      y[i] = __fadd_rn(y[i], c.bias);
  }
  if (STORE == kSilu || (STORE == kEither && p.silu_pairs)) {   // (gate, up) are neighbouring lanes: of two rows the even lane takes the first, the odd one the second
    const bool odd = c.n & 1;
    float *dst = p.C + (int64_t)m * p.ldc + (c.n >> 1) + (odd ? p.ldc : 0);
    float d[N / 2];
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float other = __shfl_xor_sync(0xffffffffu, odd ? y[i] : y[i + 1], 1);
      y[i] = odd ? other : y[i];
      y[i + 1] = odd ? y[i + 1] : other;
      d[i / 2] = 1.0f + expf(-y[i]);   // of all rows before the first reciprocal, whose branch for other ranges parts the rows' chains
    }
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float v = silu_of(y[i], y[i + 1], d[i / 2]);
      if (c.in && (ALL || (live >> (odd ? i + 1 : i) & 1)))
        *dst = v;
      dst += 2 * p.ldc;
    }
  } else {
    float *dst = p.C + (int64_t)m * p.ldc + c.n;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (c.in && (ALL || (live >> i & 1)))
        *dst = p.residual ? __fadd_rn(res[i], y[i]) : y[i];
      dst += p.ldc;
    }
  }
}
template <int STORE, int N>
__device__ __forceinline__ void load_residual(const GemmParams &p, const Channel &c, int m, int rows, float (&res)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
    res[i] = 0.f;
  if (STORE != kSilu && p.residual != nullptr) {
    const float *src = p.residual + (int64_t)m * p.ldr + c.n;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (c.in && i < rows)
        res[i] = src[(int64_t)i * p.ldr];
  }
}
// The digits' sums of N rows, ND columns each, added up.
template <int ND, int N> __device__ __forceinline__ void add_digits(const uint32_t *v, float (&y)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if constexpr (ND == 1) {
      y[i] = __uint_as_float(v[i]);
    } else {
#pragma unroll
      for (int d = 0; d < ND; ++d) {   // the digits' weights: 2^16, 2^8, 1, 2^-7, 2^-15, 2^-23
        const float b = __int2float_rn((int)v[i * ND + d]) * __uint_as_float((uint32_t)(127 + 16 - 8 * d + (d >= kPlanes)) << 23);
        y[i] = d == 0 ? b : y[i] + b;
      }
    }
  }
}
__device__ __forceinline__ void release_accumulator(uint32_t bar) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if ((threadIdx.x & 31) == 0)
    cluster_arrive(bar);
}
// Split k: a CTA's sums of row r of the tile go to the CTA of the cluster that completes the row, [split][its rows][128 channels].
struct Shares {
  uint32_t base;   // this lane's channel of this CTA's share
  uint32_t rank;   // the cluster's CTA with the same channels and the first share of k
};
__device__ __forceinline__ void give_row(const GemmParams &p, const Shares &sh, int row, float v) {
  const int to = row / p.share_rows;
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(in_cta(sh.base + (uint32_t)(row - to * p.share_rows) * (BM * 4), sh.rank + to * 2)), "f"(v)
               : "memory");
}
// The pass over all rows of a tile.  Split k: the sums go to the CTAs that complete the rows.  wait: until the accumulator at tmem is
// complete; what the first rows need from memory is requested before it.
// WIDE: some of the rows are wide, and left to the passes with six digits.
template <bool PLANES, int STORE, bool SPLIT, bool WIDE, typename Wait>
__device__ __forceinline__ void store_tile(const GemmParams &p, const Tile &t, const Channel &c, const RowScales &scales, uint32_t tmem,
                                           uint32_t release, const Shares &sh, Wait wait) {
  constexpr int ND = PLANES ? kPlanes : 1;
  const int grp = (threadIdx.x - 64) >> 7;
  int r0 = grp * CR;
  float res[CR];
  if (!SPLIT)
    load_residual<STORE, CR>(p, c, t.m0 + r0, t.rows - r0, res);
  const bool ok = wait();
  if (r0 >= t.rows || !ok) {
    release_accumulator(release);
    return;
  }
#pragma unroll 1
  for (; r0 < t.rows; r0 += kGroups * CR) {
    uint32_t v[ND * CR];
#pragma unroll
    for (int q = 0; q < ND; ++q)
      if (r0 * ND + q * CR < p.nc)
        tmem_load(tmem + r0 * ND + q * CR, *reinterpret_cast<uint32_t(*)[CR]>(v + q * CR));
    const float rs = PLANES ? scales.at(r0) : scales.v[0];
    const int left = t.rows - r0;
    uint32_t live = left >= CR ? (1u << CR) - 1 : (1u << left) - 1;
    if (WIDE)
      live &= ~(__ballot_sync(0xffffffffu, signbit(rs)) >> (r0 & 31));
    float next[CR], y[CR];
    if (!SPLIT)
      load_residual<STORE, CR>(p, c, t.m0 + r0 + kGroups * CR, left - kGroups * CR, next);
    tmem_wait_load();
    if (left <= kGroups * CR)
      release_accumulator(release);
    add_digits<ND, CR>(v, y);
    if (SPLIT) {
#pragma unroll
      for (int i = 0; i < CR; ++i)
        if (live >> i & 1)
          give_row(p, sh, r0 + i, y[i]);
    } else {
      if (live == (1u << CR) - 1)
        finish_rows<PLANES, STORE, true, CR>(p, c, t.m0 + r0, y, rs, r0 & 31, live, res);
      else
        finish_rows<PLANES, STORE, false, CR>(p, c, t.m0 + r0, y, rs, r0 & 31, live, res);
#pragma unroll
      for (int i = 0; i < CR; ++i)
        res[i] = next[i];
    }
  }
}
// The pass with six digits over `rows` rows of a tile, `first` the first: its wide rows.
template <int STORE, bool SPLIT, typename Wait>
__device__ __forceinline__ void store_wide_pass(const GemmParams &p, int m0, const Channel &c, uint32_t tmem, int first, int rows,
                                                uint32_t release, const Shares &sh, Wait wait) {
  constexpr int N = CR / 2;
  const int lane = threadIdx.x & 31, grp = (threadIdx.x - 64) >> 7;
  float rs, res[N];
  auto request = [&](int r0, float &s, float (&r)[N]) {
    s = lane < N && r0 + lane < rows ? __ldcg(p.row_scale + m0 + first + r0 + lane) : 0.f;
    if (!SPLIT)
      load_residual<STORE, N>(p, c, m0 + first + r0, rows - r0, r);
  };
  request(grp * N, rs, res);
  const bool ok = wait();
  if (grp * N >= rows || !ok) {
    release_accumulator(release);
    return;
  }
#pragma unroll 1
  for (int r0 = grp * N; r0 < rows; r0 += kGroups * N) {
    uint32_t v[kWidePlanes * N];
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (r0 * kWidePlanes + q * CR < p.nc)
        tmem_load(tmem + r0 * kWidePlanes + q * CR, *reinterpret_cast<uint32_t(*)[CR]>(v + q * CR));
    const uint32_t live = __ballot_sync(0xffffffffu, signbit(rs));
    float next_rs, next[N], y[N];
    request(r0 + kGroups * N, next_rs, next);
    tmem_wait_load();
    if (r0 + kGroups * N >= rows)
      release_accumulator(release);
    add_digits<kWidePlanes, N>(v, y);
    if (SPLIT) {
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (live >> i & 1)
          give_row(p, sh, first + r0 + i, y[i]);
    } else {
      finish_rows<true, STORE, false, N>(p, c, m0 + first + r0, y, rs, 0, live, res);
#pragma unroll
      for (int i = 0; i < N; ++i)
        res[i] = next[i];
    }
    rs = next_rs;
  }
}
// The rows that this CTA completes, shares added in order.  sums: this lane's channel of the first share.
template <bool PLANES, int STORE>
__device__ __forceinline__ void add_shares(const GemmParams &p, int m0, int rows, const Channel &c, const float *sums) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int r0 = ((threadIdx.x - 64) >> 7) * CR; r0 < rows; r0 += kGroups * CR) {
    const int m = m0 + r0, live = min(CR, rows - r0);
    float rs = 0.f, res[CR], y[CR];
    if (!PLANES)
      rs = p.row_scale[0];
    else if (lane < live)
      rs = __ldcg(p.row_scale + m + lane);
    load_residual<STORE, CR>(p, c, m, live, res);
#pragma unroll
    for (int i = 0; i < CR; ++i)
      y[i] = 0.f;
#pragma unroll 1
    for (int z = 0; z < p.splits; ++z)
#pragma unroll
      for (int i = 0; i < CR; ++i)
        if (i < live) {
          const float b = sums[(z * p.share_rows + r0 + i) * BM];
          y[i] = PLANES ? y[i] + b : __int_as_float(__float_as_int(y[i]) + __float_as_int(b));
        }
    finish_rows<PLANES, STORE, false, CR>(p, c, m, y, rs, 0, (1u << live) - 1, res);
  }
}
// mbar_wait, and what the cluster's other CTAs stored before they arrived is visible.
__device__ __forceinline__ bool wait_shares(uint64_t *bar, volatile int *ab, int *err, int code) {
  if (!mbar_wait(bar, 0, ab, err, code))
    return false;
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  return true;
}

// An epilogue warp's way through the tiles from w on; n: accumulators so far.  WIDE = false: up to a tile with wide rows.
template <bool PLANES, int STORE, bool SPLIT, bool WIDE>
__device__ __forceinline__ int epilogue(const GemmParams &p, Bars &bars, float *sums, uint32_t tmem, int w, int step, int &n) {
  const int lane = threadIdx.x & 31, quad = threadIdx.x >> 5 & 3, crank = (int)cluster_rank(), rank = crank & 1;
  const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
  const int channel = quad * 32 + lane;
  volatile int *ab = &bars.abort_flag;
  bool ok = true;
  if (w >= p.tiles)
    return w;
  RowScales scales;
  auto request = [&](const Tile &i) {
    if (PLANES)
      scales.load(p, i.m0, i.rows);
    else
      scales.v[0] = __ldcg(p.row_scale);
  };
  Tile t = tile_at(p, w);
  Channel c(p, t.n0 + rank * BM + channel);
  request(t);
#pragma unroll 1
  for (;;) {   // (a warp that gave up goes on without waiting: the barriers keep their count)
    const uint32_t wide = PLANES ? scales.wide_halves(p) : 0u;
    if (!WIDE && wide != 0)
      return w;
    const int z = crank >> 1;
    const Shares sh{smem_u32(sums + z * p.share_rows * BM + channel), (uint32_t)rank};
    auto wait = [&] {
      ok = ok && __all_sync(0xffffffffu, mbar_wait(&bars.acc_full[n & 1], n >> 1 & 1, ab, p.error, 703));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    auto release = [&] { return in_cta(smem_u32(&bars.acc_empty[n & 1]), crank & ~1); };
    store_tile<PLANES, STORE, SPLIT, WIDE>(p, t, c, scales, lanes + (n & 1) * (p.cols >> 1), release(), sh, wait);
    ++n;
    if constexpr (WIDE) {
      const int half = (p.rows + 1) >> 1;
#pragma unroll 1
      for (int h = 0; h < 2; ++h)
        if (wide >> h & 1) {
          store_wide_pass<STORE, SPLIT>(p, t.m0, c, lanes + (n & 1) * (p.cols >> 1), h * half, min(half, t.rows - h * half), release(), sh, wait);
          ++n;
        }
    }
    if constexpr (SPLIT) {
      __syncwarp();
      if (lane < p.splits)   // (release: this warp's stores come first)
        cluster_arrive(in_cta(smem_u32(&bars.sums), lane * 2 + rank));
      ok = __all_sync(0xffffffffu, wait_shares(&bars.sums, ab, p.error, 705)) && ok;
      const int row = z * p.share_rows;
      if (ok)
        add_shares<PLANES, STORE>(p, t.m0 + row, min(p.share_rows, t.rows - row), c, sums + channel);
    }
    w += step;
    if (w >= p.tiles)
      return w;
    t = tile_at(p, w);   // what it needs is on its way while the tile's products are made
    c = Channel(p, t.n0 + rank * BM + channel);
    request(t);
  }
}
// The tiles from a wide one on, as a function with a copy of the parameters (behind a generic pointer they are loaded again after every
// store: 1024 x 17920 x 1536 with one wide row 112 us, 94 with the copy).  Where a pair has many products to make (TURNS) this is part of
// the kernel, so that tiles after a wide one are as quick as those before: 84 us.  Inline everywhere it would lengthen every launch without
// a wide row: a pass of 100 rows of the 1.5B model 2.36 / 2.40 ms.
template <int STORE, bool SPLIT>
__device__ __noinline__ void epilogue_last(const GemmParams &p_in, Bars &bars, float *sums, uint32_t tmem, int w, int step, int n) {
  const GemmParams p = p_in;
  epilogue<true, STORE, SPLIT, true>(p, bars, sums, tmem, w, step, n);
}

template <bool PLANES, int STORE, bool SPLIT, bool TURNS>
__global__ void __launch_bounds__(kThreads, 1)
gemm_i8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_x) {
  constexpr int ND = PLANES ? kPlanes : 1;
  extern __shared__ __align__(1024) uint8_t smem[];
  // 1024-byte alignment of every swizzled tile
  uint8_t *tiles = reinterpret_cast<uint8_t *>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  const uint32_t stage_bytes = kWBytes + (uint32_t)(p.nc / 2) * BK;
  const int S = p.stages;
  float *sums = reinterpret_cast<float *>(tiles + S * stage_bytes);   // split k: [splits][share_rows][128]
  Bars &bars = *reinterpret_cast<Bars *>(sums + (SPLIT ? p.splits * p.share_rows * BM : 0));
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // a cluster: `splits` pairs, each with a share of the k blocks
  const int crank = (int)cluster_rank(), rank = crank & 1, z = crank >> 1;
  const int first = blockIdx.x / (2 * p.splits), step = gridDim.x / (2 * p.splits);
  const int all_blocks = (p.K + BK - 1) / BK;
  const int kb0 = all_blocks * z / p.splits, nkb = all_blocks * (z + 1) / p.splits - kb0;
  volatile int *ab = &bars.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bars.acc_full[a], 1);
      mbar_init(&bars.acc_empty[a], 2 * kEpiWarps);
    }
    mbar_init(&bars.sums, p.splits * kEpiWarps);
    bars.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {   // tensor memory: one warp (of each CTA) allocates, the same warp frees
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem_base)), "r"(p.cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  sync_cluster();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars.tmem_base, 0);
  kernel_go();   // not before the allocation: see tensor_core.cuh

  if (warp == 0) {
    // ---- loader --------------------------------------------------------------------------------------------------
    const uint32_t base = smem_u32(tiles);
    int s = 0, parity = 1;   // (waiting for the phase before a barrier's first ends at once)
    auto full = [&](int st) { return in_cta(smem_u32(&bars.full[st]), crank & ~1); };
    auto load_w = [&](const Tile &t, int i, int st) {
      if (rank == 0)
        mbar_expect_tx(&bars.full[st], 2 * stage_bytes);
      tma_load_2d(base + st * stage_bytes, &map_w, (kb0 + i) * BK, t.n0 + rank * BM, full(st));
    };
    Tile t = tile_at(p, first);
    const int ahead = min(S, nkb);
    if (lane == 0) {
      // few rows: the weights' way from memory is the GEMM; all of this CTA's share starts for L2 while the kernels before run
      // (if it has one tile: 24 x 151936 x 1536, in several turns, took 68 us with it and 60 without)
      if (p.m_tiles <= 2 && p.tiles <= step)
        for (int i = S; i < nkb; ++i)
          tma_prefetch_2d(&map_w, (kb0 + i) * BK, t.n0 + rank * BM);
      for (int i = 0; i < ahead; ++i)   // the weights do not wait for the kernel before
        load_w(t, i, i);
    }
    kernel_wait();
    RowScales scales;
    if (PLANES)
      scales.load(p, t.m0, t.rows);
    uint32_t wide = PLANES ? scales.wide_halves(p) : 0u;
    int ready = ahead;   // stages whose weights are on their way
    bool ok = true;
    for (int w = first; w < p.tiles && ok; w += step) {
      const Tile next = tile_at(p, min(w + step, p.tiles - 1));
      if (PLANES)
        scales.load(p, next.m0, next.rows);
      for (int pass = 0; pass < 3 && ok; ++pass) {
        if (pass > 0 && !(wide >> (pass - 1) & 1))
          continue;
        const CUtensorMap *map = pass ? &map_x : &map_a;
        const int y = (pass ? kWidePlanes * (t.m0 + (pass - 1) * ((p.rows + 1) >> 1)) : ND * t.m0) + rank * (p.nc / 2);
        if (lane == 0)
          for (int i = 0; i < nkb; ++i) {
            if (ready > 0) {
              --ready;
            } else {
              if (!mbar_wait(&bars.empty[s], parity, ab, p.error, 701)) {
                ok = false;
                break;
              }
              load_w(t, i, s);
            }
            tma_load_2d(base + s * stage_bytes + kWBytes, map, (kb0 + i) * BK, y, full(s));
            if (++s == S) {
              s = 0;
              parity ^= 1;
            }
          }
        ok = __all_sync(0xffffffffu, ok);
      }
      t = next;
      wide = PLANES ? scales.wide_halves(p) : 0u;
    }
  } else if (warp == 1) {
    // ---- tensor core issue (of the pair's first CTA) ------------------------------------------------------------------
    if (rank == 0) {
      kernel_wait();
      uint32_t leader;
      asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(leader));
      const uint32_t idesc = mma_desc(p.nc);
      const uint64_t d0 = smem_desc(smem_u32(tiles));
      int s = 0, parity = 0, n = 0;   // n: accumulators so far
      bool ok = true;
      Tile t = tile_at(p, first);
      RowScales scales;
      if (PLANES)
        scales.load(p, t.m0, t.rows);
      uint32_t wide = PLANES ? scales.wide_halves(p) : 0u;
      for (int w = first; w < p.tiles && ok; w += step) {
        const Tile next = tile_at(p, min(w + step, p.tiles - 1));
        if (PLANES)
          scales.load(p, next.m0, next.rows);
        for (int pass = 0; pass < 3 && ok; ++pass) {
          if (pass > 0 && !(wide >> (pass - 1) & 1))
            continue;
          ok = __all_sync(0xffffffffu, mbar_wait(&bars.acc_empty[n & 1], (n >> 1 & 1) ^ 1, ab, p.error, 704));
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t acc = tmem + (n & 1) * (p.cols >> 1);
          for (int i = 0; i < nkb && ok; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait(&bars.full[s], parity, ab, p.error, 702));
            if (!ok)
              break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t dw = d0 + ((s * stage_bytes) >> 4), dx = dw + (kWBytes >> 4);
#pragma unroll
            for (int k = 0; k < BK / 32; ++k)   // 32 int8 = 32 bytes along the swizzled row
              mma_i8(leader, acc, dw + k * 2, dx + k * 2, idesc, (i | k) != 0);
            if (leader)
              commit(&bars.empty[s]);   // arrives when the MMAs above have read the stage
            if (++s == S) {
              s = 0;
              parity ^= 1;
            }
          }
          if (ok && leader)
            commit(&bars.acc_full[n & 1]);
          ++n;
        }
        t = next;
        wide = PLANES ? scales.wide_halves(p) : 0u;
      }
    }
  } else {
    // ---- epilogue ----------------------------------------------------------------------------------------------------
    kernel_wait();   // row scales
    int n = 0, w = first;
    w = epilogue<PLANES, STORE, SPLIT, false>(p, bars, sums, tmem, w, step, n);
    if (PLANES && w < p.tiles) {
      if constexpr (TURNS)
        epilogue<true, STORE, SPLIT, true>(p, bars, sums, tmem, w, step, n);
      else
        p.silu_pairs ? epilogue_last<kSilu, SPLIT>(p, bars, sums, tmem, w, step, n) : epilogue_last<kPlain, SPLIT>(p, bars, sums, tmem, w, step, n);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  sync_cluster();   // none ends while another may still signal it
  if (warp == 1) {
    if (*ab) {   // copies of an abandoned tile may still be in flight: let them land before the CTA ends
      const unsigned long long t0 = now_ns();
      while (now_ns() - t0 < 2000000ull) {
      }
    }
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.cols) : "memory");
  }
}

// The first kernel of a call.  The GEMM behind it loads weights before it waits, so nothing but this kernel's own wait keeps
// those loads behind what the caller's stream did before: the weights may be the output of the kernel just before the call.
// Inside a session's pass the weights were there before the pass began, and the next kernel may start at once (in_pass).
__device__ __forceinline__ void chain_start(int in_pass) {
  if (in_pass)
    kernel_go();
  kernel_wait();
  if (!in_pass)
    kernel_go();
}

// ---- the A operand ------------------------------------------------------------------------------------------------------
// Four consecutive activations from k on (K is a multiple of 64; vec: 16-byte loads are possible).
__device__ __forceinline__ float4 load4(const float *row, int k, bool vec) {
  if (vec)
    return __ldg(reinterpret_cast<const float4 *>(row + k));
  return make_float4(row[k], row[k + 1], row[k + 2], row[k + 3]);
}
// First k of group j of 16-byte unit u of a packed row: units lie in blocks of 32 (the last block may be shorter).
__device__ __forceinline__ int unit_k(int u, int j, int units) {
  const int b = u >> 5, nu = min(32, units - 32 * b);
  return b * 512 + j * (nu * 4) + 4 * (u & 31);
}

// A row's fixed-point scale, from the bit pattern of its largest magnitude: |X| <= 0x7F7F7F, what three signed digits hold (a
// magnitude whose mantissa would round beyond that takes the next power of two).  *inv undoes it; NaN for a row with an infinity
// or a NaN.  Below 2^-104 the scale stays, and six digits reach down to the smallest subnormal.
__device__ __forceinline__ float plane_scale(uint32_t absbits, float *inv) {
  const int e = max((int)((absbits + 0x10102u) >> 23) - 127, -104);
  *inv = absbits >= 0x7f800000u ? __uint_as_float(0x7fffffffu) : __uint_as_float((uint32_t)(e - 22 + 127) << 23);
  return __uint_as_float((uint32_t)(22 - e + 127) << 23);
}

// A[M,K] f32 -> planes [M][3][K] int8 in the k order of the packed weight rows, and the rows' scales (the sign says that a row is
// wide); optional RMSNorm of every row (the factor 1/rms goes into the scale).  T threads per row, a thread takes 16-byte
// units: it reads four groups of four k and writes whole 16-byte pieces of the planes.  The row is read once and stays in
// registers up to 48 T elements.  Outside a pass it also clears the call's error word (head).
//
// Wide rows.  Rounding to a unit leaves 0.29 units (rms) in every element, which must be no more than the 2^-19 of an element
// that two bf16 terms leave: the row's bulk has to have an rms of at least 2^17 units.  Its bulk is what lies below a quarter of
// the largest magnitude, and is also to have a mean of 2^16, so that a few percent of large elements do not pass for bulk.  A
// row with channels more than about 32 times the rest misses that, and is written a second time, into `wides` [M][6][K]: three
// more digits, of what the first three leave over in units of 2^-23, exact down to
// 2^-45 of the largest magnitude.  One sum decides for nearly all other rows: a mean magnitude of 2^17.5 units.
constexpr int kUnits = 3;
__global__ void __launch_bounds__(256)
planes_kernel(const float *A, int64_t lda, int M, int K, const float *norm_w, float eps, int T, int vec, uint8_t *planes,
              float *row_scale, uint32_t *head, int head_words, int in_pass, uint8_t *wides) {
  chain_start(in_pass);
  __shared__ uint32_t s_mx[8];
  __shared__ float s_ss[8], s_s1[8], s_bulk[8][3];
  const int t = threadIdx.x % T, m = blockIdx.x * (256 / T) + threadIdx.x / T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < head_words; i += 256)
      head[i] = 0u;
  const int units = K >> 4, step = kUnits * T;
  const float *row = A + (int64_t)min(m, M - 1) * lda;
  float4 v[kUnits][4];
  auto load = [&](int u0) {
#pragma unroll
    for (int i = 0; i < kUnits; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int u = u0 + t + i * T;
        v[i][j] = u < units ? load4(row, unit_k(u, j, units), vec) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
  };
  float ss = 0.f, s1 = 0.f;
  uint32_t mx = 0;
  auto weigh = [&](int u0, bool stats) {   // times the norm weight
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
      const int u = u0 + t + i * T;
      if (u < units)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float4 &x = v[i][j];
          if (norm_w != nullptr) {
            if (stats)
              ss = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, ss))));
            const float4 w = load4(norm_w, unit_k(u, j, units), vec);
            x = make_float4(x.x * w.x, x.y * w.y, x.z * w.z, x.w * w.w);
          }
          const uint32_t a = 0x7fffffffu;
          mx = max(mx, max(max(__float_as_uint(x.x) & a, __float_as_uint(x.y) & a),
                           max(__float_as_uint(x.z) & a, __float_as_uint(x.w) & a)));
          if (stats)
            s1 += (fabsf(x.x) + fabsf(x.y)) + (fabsf(x.z) + fabsf(x.w));
        }
    }
  };
  for (int u0 = 0; u0 < units; u0 += step) {
    load(u0);
    weigh(u0, true);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  ss = warp_sum(ss);
  s1 = warp_sum(s1);
  const int w0 = (threadIdx.x / T) * (T / 32);   // the row's first warp
  if (T > 32) {
    if (lane == 0) {
      s_mx[warp] = mx;
      s_ss[warp] = ss;
      s_s1[warp] = s1;
    }
    __syncthreads();
    mx = 0;
    ss = s1 = 0.f;
    for (int w = 0; w < T / 32; ++w) {
      mx = max(mx, s_mx[w0 + w]);
      ss += s_ss[w0 + w];
      s1 += s_s1[w0 + w];
    }
  }
  if (m >= M)
    return;
  float inv;
  const float scale = plane_scale(mx, &inv);
  bool wide = false;
  if (mx != 0u && mx < 0x7f800000u && !(s1 < 3e38f && s1 * scale >= 185364.f * (float)K)) {
    float bulk2 = 0.f, bulk = 0.f;   // of |X|
    const float cut = __uint_as_float(mx) * scale * 0.25f;
    auto add = [&](float v) {
      const float X = fabsf(v * scale);
      if (X <= cut) {
        bulk2 = fmaf(X, X, bulk2);
        bulk += X;
      }
    };
    for (int u0 = 0; u0 < units; u0 += step) {
      if (units > step) {
        load(u0);
        weigh(u0, false);
      }
#pragma unroll
      for (int i = 0; i < kUnits; ++i)   // (units beyond the row are zero)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          add(v[i][j].x);
          add(v[i][j].y);
          add(v[i][j].z);
          add(v[i][j].w);
        }
    }
    auto over_row = [&](float a, int at) {   // a summed over the row's threads
      a = warp_sum(a);
      if (T > 32) {
        if (lane == 0)
          s_bulk[warp][at] = a;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / T), "r"(T) : "memory");   // the row's threads
        a = 0.f;
        for (int w = 0; w < T / 32; ++w)
          a += s_bulk[w0 + w][at];
      }
      return a;
    };
    bulk2 = over_row(bulk2, 0);
    if (!(bulk2 >= 17179869184.f * (float)K) || !(over_row(bulk, 1) >= 65536.f * (float)K)) {
      float rest = 0.f;   // what rounding leaves over: a row without is exact as it is
#pragma unroll 1
      for (int k = 4 * t; k < K; k += 4 * T) {
        float4 x = load4(row, k, vec);
        if (norm_w != nullptr) {
          const float4 n = load4(norm_w, k, vec);
          x = make_float4(x.x * n.x, x.y * n.y, x.z * n.z, x.w * n.w);
        }
        auto left = [&](float a) { return fabsf(a * scale - rintf(a * scale)); };
        rest += (left(x.x) + left(x.y)) + (left(x.z) + left(x.w));
      }
      wide = over_row(rest, 2) > 0.f;
    }
  }
  if (t == 0) {
    const float rs = norm_w != nullptr ? inv * rsqrtf(ss * (1.0f / (float)K) + eps) : inv;
    row_scale[m] = __uint_as_float((__float_as_uint(rs) & 0x7fffffffu) | (wide ? 0x80000000u : 0u));
  }
  uint8_t *dst = planes + (int64_t)m * kPlanes * K, *wdst = wides + (int64_t)m * kWidePlanes * K;
  for (int u0 = 0; u0 < units; u0 += step) {
    if (units > step) {
      load(u0);
      weigh(u0, false);
    }
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
      const int u = u0 + t + i * T;
      if (u < units) {
        uint32_t w[4][4];   // [group][plane]
#pragma unroll
        for (int j = 0; j < 4; ++j)
          plane_words(fixed_digits(v[i][j].x, scale), fixed_digits(v[i][j].y, scale), fixed_digits(v[i][j].z, scale),
                      fixed_digits(v[i][j].w, scale), w[j]);
#pragma unroll
        for (int pl = 0; pl < kPlanes; ++pl)   // (the digit of 2^24 is zero)
          *reinterpret_cast<uint4 *>(dst + (int64_t)pl * K + u * 16) =
              make_uint4(w[0][pl + 1], w[1][pl + 1], w[2][pl + 1], w[3][pl + 1]);
      }
    }
  }
  if (!wide)
    return;
#pragma unroll 1
  for (int u = t; u < units; u += T) {   // from memory again: few registers
    uint32_t w[4][4], l[4][4];
    auto rest = [&](float x) { return fixed_digits(x * scale - rintf(x * scale), 8388608.f); };   // exact, |rest| <= 2^22
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float4 x = load4(row, unit_k(u, j, units), vec);
      if (norm_w != nullptr) {
        const float4 n = load4(norm_w, unit_k(u, j, units), vec);
        x = make_float4(x.x * n.x, x.y * n.y, x.z * n.z, x.w * n.w);
      }
      plane_words(fixed_digits(x.x, scale), fixed_digits(x.y, scale), fixed_digits(x.z, scale), fixed_digits(x.w, scale), w[j]);
      plane_words(rest(x.x), rest(x.y), rest(x.z), rest(x.w), l[j]);
    }
#pragma unroll
    for (int pl = 0; pl < kPlanes; ++pl) {
      uint4 *at = reinterpret_cast<uint4 *>(wdst + (int64_t)pl * K + u * 16);
      *at = make_uint4(w[0][pl + 1], w[1][pl + 1], w[2][pl + 1], w[3][pl + 1]);
      *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(at) + (int64_t)kPlanes * K) =
          make_uint4(l[0][pl + 1], l[1][pl + 1], l[2][pl + 1], l[3][pl + 1]);
    }
  }
}

// ---- W8A8: one dynamic scale for the whole activation tensor -------------------------------------------------------------
// buddy-mlir's QuantizedMatmulOp (frontend/Python/ops/linalg.py:12728-12846): s = max(absmax / 127, 1e-10),
// q = clamp(rne(x * (1 / s)), -128, 127), an exact i8 x i8 -> i32 contraction, y = float(acc) * (s * weight_scale[n])
// (+ bias).  Every step is reproduced operation by operation, so the result is bit-identical to the reference arithmetic.
constexpr int kMaxParts = 256;   // partial maxima, in the workspace head

// max |x| of every CTA's share of the tensor (non-negative floats order like their bit patterns); clears the call's
// error word (null in a pass: the word collects what any of its GEMMs leaves).
__global__ void __launch_bounds__(256)
absmax_kernel(const float *A, int64_t lda, int M, int K, int vec, uint32_t *part, uint32_t *head, int head_words,
              int in_pass) {
  chain_start(in_pass);
  __shared__ uint32_t s_mx[8];
  if (blockIdx.x == 0 && (int)threadIdx.x < head_words)
    head[threadIdx.x] = 0u;
  float fm = 0.f;
  const int k4 = K >> 2;
  const int64_t total = (int64_t)M * k4, stride = (int64_t)gridDim.x * 256;
  for (int64_t i0 = (int64_t)blockIdx.x * 256 + threadIdx.x; i0 < total; i0 += 4 * stride) {
    float4 v[4];   // four loads in flight
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = min(i0 + u * stride, total - 1);
      const uint32_t m = (uint32_t)i / (uint32_t)k4;   // M * K < 2^33
      v[u] = load4(A + (int64_t)m * lda, (int)(i - (int64_t)m * k4) * 4, vec);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      fm = fmaxf(fmaxf(fm, fmaxf(fabsf(v[u].x), fabsf(v[u].y))), fmaxf(fabsf(v[u].z), fabsf(v[u].w)));
  }
  uint32_t mx = __reduce_max_sync(0xffffffffu, __float_as_uint(fm));
  if ((threadIdx.x & 31) == 0)
    s_mx[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w)
      mx = max(mx, s_mx[w]);
    part[blockIdx.x] = mx;
  }
}

// A 16-byte unit per thread, in the k order of the packed weight rows; CTA 0 also leaves the scale for the epilogue.
__global__ void __launch_bounds__(256)
quantize_kernel(const float *A, int64_t lda, int M, int K, int vec, const uint32_t *part, int parts, float *scale_out,
                uint8_t *q) {
  kernel_go();   // absmax_kernel, before it, has waited as the call requires
  kernel_wait();
  __shared__ uint32_t s_mx[8];
  uint32_t mx = threadIdx.x < parts ? __ldcg(part + threadIdx.x) : 0u;
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0)
    s_mx[threadIdx.x >> 5] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w)
    mx = max(mx, s_mx[w]);
  const float scale = fmaxf(__fmul_rn(__uint_as_float(mx), __fdiv_rn(1.0f, 127.0f)), 1e-10f);
  const float inv = __fdiv_rn(1.0f, scale);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *scale_out = scale;
  const int units = K >> 4;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (int64_t)M * units)
    return;
  const int m = (int)(i / units), u = (int)(i - (int64_t)m * units);
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 v = load4(A + (int64_t)m * lda, unit_k(u, j, units), vec);
    const float x[4] = {v.x, v.y, v.z, v.w};
    w[j] = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float r = rintf(__fmul_rn(x[e], inv));     // the f32 -> i32 cast rounds to nearest even
      w[j] |= ((uint32_t)(int)fminf(fmaxf(r, -128.0f), 127.0f) & 0xFFu) << (8 * e);
    }
  }
  *reinterpret_cast<uint4 *>(q + (int64_t)m * K + u * 16) = make_uint4(w[0], w[1], w[2], w[3]);
}

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  return fn;
}

int make_map(CUtensorMap *map, CUtensorMapDataType dt, int bk, void *base, uint64_t inner, uint64_t rows,
             uint64_t pitch_bytes, CUtensorMapSwizzle swz, int box_rows = 128) {
  EncodeFn fn = encode_fn();
  if (!fn)
    return fail(B200_ECUDA, "gemm_w8: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {inner, rows};
  const cuuint64_t strides[1] = {pitch_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)bk, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult rc = fn(map, dt, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS)
    return fail(B200_ECUDA, "gemm_w8: cuTensorMapEncodeTiled failed (%d)", (int)rc);
  return B200_OK;
}

// How a GEMM is laid over the chip's 74 pairs of SMs.
struct Plan {
  int nc, rows, m_tiles, tiles, splits, share_rows, stages, grid, cols, smem;
};
constexpr int kMostShared = 198 * 1024;

// Costs in clocks.  A k block costs a pair its products (8192 of 128 x 128 x nc a clock and SM) or its bytes (64 a clock and SM, 45
// when all pairs load), whichever takes longer; a tile's epilogue runs under the next tile's products, except the last.  Every pair that
// is taken counts: the next kernel of a pass could start there (a decode step's attention after q|k|v of 24 rows took 17 us behind
// 128 CTAs, 14 behind 16).  Sums across a cluster cost time for themselves and for their rows, which also take memory from the ring.
// Clusters of four, six and eight CTAs leave SMs over, which differ from part to part (SMs that are switched off): 33, 22 and 15 of
// them fit here, and one more than fits takes a second turn: so many shares are not taken.  Row tiles x shares of k, us, weights from
// memory, * where the clusters take two turns:
//   24 x 2048 x 1536      1 x 1  9.4    2 x 1  9.4    1 x 4  9.7        24 x 1536 x 8960      1 x 3 14.9   1 x 4 13.8
//   100 x 1536 x 8960     3 x 2 18.5    3 x 3 16.9    2 x 4 16.9        200 x 1536 x 8960     5 x 2 20.8   3 x 3 20.7   3 x 4 32.3 *
//   366 x 1536 x 8960     5 x 2 25.1    5 x 1 28.6   12 x 1 26.3        700 x 1536 x 8960    11 x 1 30.5   9 x 1 34.6  18 x 1 45.7
//   24 x 4096 x 4096      1 x 1 14.9    1 x 3 13.3    1 x 4 21.5 *      24 x 4096 x 12288     1 x 2 24.2   1 x 3 20.8   1 x 4 31.7 *
//   W8A8 366 x 1536 x 8960  4 x 2 27.0   3 x 3 28.0   2 x 4 30.6        W8A8 366 x 1536 x 1536  6 x 1 10.3  4 x 1 10.6  2 x 2 19.1
Plan make_plan(int M, int N, int K, int nd, const int (&held)[kMaxSplits + 1]) {
  const int nkb = (K + BK - 1) / BK, n_tiles = (N + 2 * BM - 1) / (2 * BM), most = nd == 1 ? 256 : 84, least_tiles = (M + most - 1) / most;
  Plan best{};
  float least = 0.f;
  for (int mt = least_tiles; mt < least_tiles + 16 && mt <= M; ++mt) {
    const int rows = (M + mt - 1) / mt, need = nd == 1 ? rows : kWidePlanes * ((rows + 1) / 2), nc = (need + 31) / 32 * 32;
    const int m_tiles = (M + rows - 1) / rows, tiles = n_tiles * m_tiles;
    for (int splits = 1; splits <= kMaxSplits && splits <= std::max(nkb / 2, 1); ++splits) {
      if (splits > 1 && tiles > held[splits])
        break;
      const float rounds = (float)((tiles + kPairs - 1) / kPairs), busy = (float)std::min(tiles * splits, kPairs);
      const float per_kb = std::max(2.f * nc, (2 * BM + nc) * (1.f + 0.4f * busy / kPairs));
      const float cost = rounds * (float)((nkb + splits - 1) / splits) * per_kb + 1000.f + 20.f * rows +
                         (splits > 1 ? 2000.f + 100.f * rows : 0.f) + 50.f * busy;
      if (best.nc == 0 || cost < least) {
        least = cost;
        best.nc = nc;
        best.rows = rows;
        best.m_tiles = m_tiles;
        best.tiles = tiles;
        best.splits = splits;
      }
    }
  }
  best.share_rows = (best.rows + best.splits - 1) / best.splits;
  const int clusters = best.splits > 1 ? best.tiles : std::min(best.tiles, kPairs), stage = (int)kWBytes + best.nc / 2 * BK;
  best.grid = clusters * 2 * best.splits;
  const int blocks = (best.tiles + clusters - 1) / clusters * ((nkb + best.splits - 1) / best.splits);
  const int extra = 1024 + (int)sizeof(Bars) + (best.splits > 1 ? best.splits * best.share_rows * BM * 4 : 0);
  best.stages = std::min({kMaxStages, blocks, (kMostShared - extra) / stage});
  best.smem = extra + best.stages * stage;
  best.cols = 32;
  while (best.cols < 2 * best.nc)
    best.cols *= 2;
  return best;
}

template <bool PLANES, int STORE, bool SPLIT, bool TURNS>
int launch_gemm(const Plan &pl, const void *a, const void *x, const void *w, GemmParams &p, cudaStream_t st) {
  CUtensorMap map_a, map_w, map_x;
  const int box = pl.nc / 2;
  if (int rc = make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, BK, const_cast<void *>(a), p.K, (uint64_t)p.M * (PLANES ? kPlanes : 1),
                        (uint64_t)p.K, CU_TENSOR_MAP_SWIZZLE_128B, box))
    return rc;
  if (int rc = make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, BK, const_cast<void *>(w), p.K, p.N, (uint64_t)p.K,
                        CU_TENSOR_MAP_SWIZZLE_128B, BM))
    return rc;
  map_x = map_a;
  if (PLANES)
    if (int rc = make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, BK, const_cast<void *>(x), p.K, (uint64_t)p.M * kWidePlanes,
                          (uint64_t)p.K, CU_TENSOR_MAP_SWIZZLE_128B, box))
      return rc;
  p.nc = pl.nc;
  p.rows = pl.rows;
  p.m_tiles = pl.m_tiles;
  p.tiles = pl.tiles;
  p.splits = pl.splits;
  p.share_rows = pl.share_rows;
  p.stages = pl.stages;
  p.cols = pl.cols;
  static RaisedOn raised;
  if (int rc = raise_shared_limit(raised, (const void *)gemm_i8_kernel<PLANES, STORE, SPLIT, TURNS>, kMostShared))
    return rc;
  return launch_after_clusters(2 * pl.splits, gemm_i8_kernel<PLANES, STORE, SPLIT, TURNS>, dim3(pl.grid), kThreads, pl.smem, st, map_a, map_w, p, map_x);
}
// How many clusters of 2 x splits CTAs the current device holds at once; negative: an error code.
int clusters_held(int splits) {
  static std::atomic<int> known[64][kMaxSplits + 1];   // per device, once it has been asked: one more than the number
  int dev = 0, n = 0;
  B200_CUDA(cudaGetDevice(&dev));
  std::atomic<int> *seen = dev >= 0 && dev < 64 ? &known[dev][splits] : nullptr;
  if (seen != nullptr && (n = seen->load(std::memory_order_relaxed)) > 0)
    return n - 1;
  static RaisedOn raised;
  auto kern = gemm_i8_kernel<true, kEither, true, false>;
  if (int rc = raise_shared_limit(raised, (const void *)kern, kMostShared))
    return rc;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kSms / (2 * splits) * 2 * splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kMostShared;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  B200_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
  if (seen != nullptr)
    seen->store(n + 1, std::memory_order_relaxed);
  return n;
}
template <bool PLANES> int launch_plan(const void *a, const void *x, const void *w, GemmParams &p, cudaStream_t st) {
  int held[kMaxSplits + 1] = {};
  for (int s = 2; s <= kMaxSplits; ++s)
    if ((held[s] = clusters_held(s)) < 0)
      return held[s];
  const Plan pl = make_plan(p.M, p.N, p.K, PLANES ? kPlanes : 1, held);
  if (pl.splits > 1)
    return launch_gemm<PLANES, kEither, true, false>(pl, a, x, w, p, st);
  // Many products: turns of the pairs times blocks of k.  us without / with one wide row, inline / as a function: 1024 x 17920 x 1536 (13 x 12)
  // 69.1 / 84 and 71.0 / 94, 1024 x 1536 x 8960 (2 x 70) 48.3 / 66 and 51.5 / 72, 366 x 17920 x 1536 (5 x 12) 30.2 / 41 and 30.8 / 43, 100 x
  // 17920 x 1536 (2 x 12) 16.7 / 24 and 16.5 / 26, 1024 x 1536 x 1536 (2 x 12) 16.4 / 22 and 16.1 / 23
  const int pairs = pl.grid / 2;
  if (PLANES && pl.tiles > pairs && (pl.tiles + pairs - 1) / pairs * ((p.K + BK - 1) / BK) >= 56)
    return p.silu_pairs ? launch_gemm<PLANES, kSilu, false, PLANES>(pl, a, x, w, p, st) : launch_gemm<PLANES, kPlain, false, PLANES>(pl, a, x, w, p, st);
  return launch_gemm<PLANES, kEither, false, false>(pl, a, x, w, p, st);
}

} // namespace

} // namespace b200

using namespace b200;

extern "C" {

int64_t b200_gemm_w8_workspace_bytes(int M, int64_t K) {
  if (M < 1 || K < 1)
    return 0;
  // head, row scales, planes, the wide rows' planes
  return kHeadBytes + (int64_t)M * 4 + 511 + (int64_t)(kPlanes + kWidePlanes) * M * packed_k(B200_W_I8, K);
}

int b200_gemm_w8(const b200_weight *w, const float *A, int M, int64_t lda, float *C, int64_t ldc,
                 const float *residual, int64_t ldr, const float *norm_weight, float norm_eps,
                 int silu_pairs, void *workspace, int64_t workspace_bytes, void *stream) {
  return b200::gemm_w8_run(w, A, M, lda, C, ldc, residual, ldr, norm_weight, norm_eps, silu_pairs, workspace, workspace_bytes,
                           false, (cudaStream_t)stream);
}

} // extern "C"

namespace b200 {
// in_pass: a call of a session's pass, whose weights no kernel of the pass writes, and whose error word the session clears when
// it reads it at the end of the pass.
int gemm_w8_run(const b200_weight *w, const float *A, int M, int64_t lda, float *C, int64_t ldc, const float *residual,
                int64_t ldr, const float *norm_weight, float norm_eps, int silu_pairs, void *workspace,
                int64_t workspace_bytes, bool in_pass, cudaStream_t st) {
  if (!w || !A || !C || !workspace)
    return fail(B200_EINVAL, "gemm_w8: null argument");
  if (w->kind != B200_W_I8 || w->scale_dtype != B200_F32 || !w->scale || !w->w)
    return fail(B200_EINVAL, "gemm_w8: int8 per-channel weights with f32 scales expected");
  if (M < 1 || w->K % 64 != 0 || w->K > 131008 || w->N < 1 || (silu_pairs && (w->N & 1)))
    return fail(B200_EINVAL, "gemm_w8: M >= 1, K a multiple of 64 up to 131008 (s32 sums), even N for gate/up pairs");
  if (((uintptr_t)w->w & 15) || ((uintptr_t)workspace & 255))
    return fail(B200_EINVAL, "gemm_w8: weight rows must be 16-byte aligned, the workspace 256-byte aligned");
  if (workspace_bytes < b200_gemm_w8_workspace_bytes(M, w->K))
    return fail(B200_EINVAL, "gemm_w8: workspace too small");
  if (int rc = ensure_device())
    return rc;
  const int K = (int)w->K, N = (int)w->N;
  char *ws = (char *)workspace;
  float *row_scale = reinterpret_cast<float *>(ws + kHeadBytes);
  uint8_t *planes = reinterpret_cast<uint8_t *>(ws + (kHeadBytes + (int64_t)M * 4 + 255) / 256 * 256);
  uint8_t *wides = planes + (int64_t)M * kPlanes * K;
  GemmParams p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.scale = (const float *)w->scale;
  p.bias = (const float *)w->bias;
  p.row_scale = row_scale;
  p.residual = silu_pairs ? nullptr : residual;   // SiLU pairs have none: the kernel would ask for N columns of it
  p.C = C;
  p.ldc = ldc;
  p.ldr = ldr;
  p.silu_pairs = silu_pairs;
  p.error = reinterpret_cast<int *>(ws);
  // threads per row: as few as keep it in registers, more when there are few rows
  int T = 32;
  while (T < 256 && (K > T * 16 * kUnits || (int64_t)M * T < kSms * 256))
    T *= 2;
  const int vec = (lda & 3) == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)norm_weight & 15) == 0;
  if (int rc = launch_after(planes_kernel, dim3((M + 256 / T - 1) / (256 / T)), 256, 0, st, A, lda, M, K, norm_weight, norm_eps, T,
                            vec, planes, row_scale, reinterpret_cast<uint32_t *>(ws),
                            in_pass ? 0 : kHeadWords, in_pass ? 1 : 0, wides))
    return rc;
  return launch_plan<true>(planes, wides, w->w, p, st);
}
} // namespace b200

extern "C" {

/* W8A8 (buddy-mlir's QuantizedMatmulOp): workspace = b200_gemm_w8a8_workspace_bytes(M, K). */
int64_t b200_gemm_w8a8_workspace_bytes(int M, int64_t K) {
  if (M < 1 || K < 1)
    return 0;
  return kHeadBytes + kMaxParts * 4 + ((int64_t)M * K + 255) / 256 * 256;
}

int b200_gemm_w8a8(const b200_weight *w, const float *A, int M, int64_t lda, float *C, int64_t ldc,
                   void *workspace, int64_t workspace_bytes, void *stream) {
  return b200::gemm_w8a8_fused(w, A, M, lda, C, ldc, nullptr, 0, 0, workspace, workspace_bytes, false,
                               (cudaStream_t)stream);
}

} // extern "C"

namespace b200 {
// b200_gemm_w8a8 with the f32 operations that follow a projection in the model folded into the
// store: residual != NULL gives C = residual + y (in place allowed), silu_pairs gives
// C[m, j] = silu(y[m, 2j]) * y[m, 2j + 1] over N / 2 columns.  The same roundings as the
// separate operations.
int gemm_w8a8_fused(const b200_weight *w, const float *A, int M, int64_t lda, float *C, int64_t ldc,
                    const float *residual, int64_t ldr, int silu_pairs, void *workspace, int64_t workspace_bytes,
                    bool in_pass, cudaStream_t st) {
  if (!w || !A || !C || !workspace)
    return fail(B200_EINVAL, "gemm_w8a8: null argument");
  if (silu_pairs && ((w->N & 1) || residual))
    return fail(B200_EINVAL, "gemm_w8a8: gate / up pairs need an even N and take no residual");
  if (w->kind != B200_W_I8 || w->scale_dtype != B200_F32 || !w->scale || !w->w)
    return fail(B200_EINVAL, "gemm_w8a8: int8 per-channel weights with f32 scales expected");
  if (M < 1 || w->K % 64 != 0 || w->N < 1)
    return fail(B200_EINVAL, "gemm_w8a8: M >= 1 and K a multiple of 64 expected");
  if (((uintptr_t)w->w & 15) || ((uintptr_t)workspace & 255))
    return fail(B200_EINVAL, "gemm_w8a8: weight rows must be 16-byte aligned, the workspace 256-byte aligned");
  if (workspace_bytes < b200_gemm_w8a8_workspace_bytes(M, w->K))
    return fail(B200_EINVAL, "gemm_w8a8: workspace too small");
  if (int rc = ensure_device())
    return rc;
  const int K = (int)w->K, N = (int)w->N;
  char *ws = (char *)workspace;
  float *act_scale = reinterpret_cast<float *>(ws) + 2;
  uint32_t *part = reinterpret_cast<uint32_t *>(ws + kHeadBytes);
  uint8_t *q = reinterpret_cast<uint8_t *>(ws + kHeadBytes + kMaxParts * 4);
  GemmParams p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.scale = (const float *)w->scale;
  p.bias = (const float *)w->bias;
  p.row_scale = act_scale;
  p.C = C;
  p.ldc = ldc;
  p.residual = residual;
  p.ldr = ldr;
  p.silu_pairs = silu_pairs;
  p.error = reinterpret_cast<int *>(ws);
  const int vec = (lda & 3) == 0 && ((uintptr_t)A & 15) == 0;
  const int parts = (int)std::min<int64_t>(((int64_t)M * K / 4 + 1023) / 1024, kMaxParts);
  if (int rc = launch_after(absmax_kernel, dim3(parts), 256, 0, st, A, lda, M, K, vec, part,
                            in_pass ? nullptr : reinterpret_cast<uint32_t *>(ws), in_pass ? 0 : kHeadWords, in_pass ? 1 : 0))
    return rc;
  const int64_t units = (int64_t)M * (K / 16);
  if (int rc = launch_after(quantize_kernel, dim3((unsigned)((units + 255) / 256)), 256, 0, st, A, lda, M, K, vec,
                            (const uint32_t *)part, parts, act_scale, q))
    return rc;
  return launch_plan<false>(q, q, w->w, p, st);
}
} // namespace b200

extern "C" {

/* 0, or the code of the first bounded wait that gave up in the last b200_gemm_w8 on this workspace
 * (reads the error word; synchronises the stream). */
int b200_gemm_w8_status(void *workspace, void *stream) {
  if (!workspace)
    return fail(B200_EINVAL, "gemm_w8_status: null workspace");
  int code = 0;
  B200_CUDA(cudaMemcpyAsync(&code, workspace, 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  B200_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  if (code != 0)
    return fail(B200_ECUDA, "gemm_w8: a bounded wait gave up (code %d)", code);
  return B200_OK;
}

} // extern "C"
