// Causal attention of many query rows (a prefill chunk) on the 5th-generation tensor cores, at f32 precision.
//
// buddy-mlir's prefill attention (frontend/Python/ops/tosa.py:14245-14252 per key, the fused form of its flash-attention
// lowering) is f32 throughout, so every operand goes to the tensor cores as three bf16 terms whose sum is the f32 value
// exactly (24 = 3 x 8 bits), and a product is six of the nine term products (the three left out are below 2^-24 of it):
// kind::f16, f32 accumulators, the small products first so that only the last D / 16 steps round at the size of the sum.
// The accumulators of a key tile are read out and added up across tiles in registers.  Measured against f64 the result is
// as close as that of f32 FMAs.
//
// Two kernels.  kv_image_kernel writes a head's K and V in tiles of 64 keys as the shared-memory images the tensor cores
// read: three planes of K [64 keys][D] and of V transposed [D][64 keys], rows of 128 bytes, 128-byte swizzle; keys are
// gathered from a contiguous cache or from pages.  prefill_attn_kernel takes 128 query vectors of a kv head (query row r / G,
// head r % G: consecutive rows share K and V) against the images: one thread copies planes (16 KB each, cp.async.bulk; four
// slots of K and three of V, given back as soon as the last of a plane's products has read it), one warp issues tcgen05.mma
// (whole-warp control flow: in a one-lane branch the operands of an instruction take longer to set up than it takes to run,
// 1.6x on the whole kernel), eight warps do the softmax.  A thread owns half the keys of a row's scores (its max goes through
// shared memory to the other half) and half the columns of its output.  S = Q K^T of the next tile runs while this tile's P
// is made: P goes back to tensor memory as the A operand of O = P V.
//
// Bound by the tensor pipe: per key tile 48 products of 64 columns (48 clocks each, measured; half the pipe's rate, but a
// wider tile of keys would not fit beside Q's three planes) and 24 of 128 (64 clocks), 3840 clocks at D = 128; softmax and
// conversion run beside it.  f32 FMAs at 128 per clock would need 16384.  1000 rows, 12 heads on 2, D = 128, a layer: 219 us
// for register-tiled FMAs, 42 here and 3.5 for the images; 366 rows 25, 64 rows 14 (with a divide per output element 45, 31 and 16).
#include "common.cuh"
#include "quotient.cuh"
#include "tensor_core.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kRows = 128;            // query vectors per CTA
constexpr int kKeys = 64;             // keys per tile: 128 bytes of a V^T row
constexpr int kTerms = 3;             // bf16 terms per f32
constexpr int kKSlots = 4;            // planes of K in shared memory: a tile's three and the next tile's first
constexpr int kSoftmaxWarps = 8;
constexpr int kThreads = (kSoftmaxWarps + 2) * 32;
constexpr float kSeed = -1.0e30f;     // of the running max
constexpr int kSms = 148;
constexpr int kMostSplits = 64;       // CTAs that share the keys of a row tile
constexpr int kMaxShares = 512;       // slots for shares: row tiles x the largest number of splits
constexpr uint32_t kColS = 0, kColP = 128, kColO = 256, kCols = 512;   // tensor memory: 2 x S, P, 2 x O

template <int D> struct Tile {
  static constexpr uint32_t Q_PLANE = kRows * D * 2, K_PLANE = kKeys * D * 2;
  static constexpr uint32_t Q_BYTES = kTerms * Q_PLANE, KV_BYTES = kTerms * K_PLANE;
  static constexpr int LDO = D + 4;                             // output rows staged over the K and V tiles
  static constexpr int PART = kRows * (D + 2);                  // a share of a row tile, in floats
  static_assert(kRows * LDO * 4 <= (kKSlots + kTerms) * (int)K_PLANE, "the staged output fits");
  static constexpr uint32_t K_RING = kKSlots * K_PLANE, V_RING = kTerms * K_PLANE;
  static constexpr int SMEM = 1024 + Q_BYTES + K_RING + V_RING + 4096;
};

struct Bars {
  uint64_t k_full[kKSlots], k_empty[kKSlots], v_full[kTerms], v_empty[kTerms], s_full[2], p_ready, o_full[2];
  uint32_t tmem_base;
  int abort_flag, last;
  float mx[2][2][kRows];   // [tile parity][half of the keys][row]
  float sum[2][kRows];
};
static_assert(sizeof(Bars) <= 4096, "");

// v = t[0] + t[1] + t[2], two values at a time (the first in the low half)
__device__ __forceinline__ uint32_t take_bf16(float &a, float &b) {
  uint32_t w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(b), "f"(a));
  a -= __uint_as_float(w << 16);
  b -= __uint_as_float(w & 0xffff0000u);
  return w;
}
__device__ __forceinline__ void split8(float (&v)[8], uint4 (&t)[kTerms]) {
#pragma unroll
  for (int q = 0; q < kTerms; ++q)
    t[q] = make_uint4(take_bf16(v[0], v[1]), take_bf16(v[2], v[3]), take_bf16(v[4], v[5]), take_bf16(v[6], v[7]));
}
// byte offset of 16-byte chunk c of row r in a tile of 128-byte rows, 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// grid (key tiles, kv heads, 2 x parts): a part of the tile's K (z even) or V (odd), 8 values per thread.  Keys from
// n_keys on are zero.
template <int D>
__global__ void __launch_bounds__(256)
kv_image_kernel(const float *kc, const float *vc, int max_len, int n_keys, const int32_t *table, int page, uint8_t *images,
                uint32_t *arrived, int counters) {
  kernel_wait();
  kernel_go();   // not before: the next kernel reads Q, which the kernel before this one writes, without waiting
  if (blockIdx.x + blockIdx.y + blockIdx.z == 0)
    for (int i = threadIdx.x; i < counters; i += 256)
      arrived[i] = 0u;
  using T = Tile<D>;
  const int k0 = blockIdx.x * kKeys, hk = blockIdx.y, kv_heads = gridDim.y;
  uint8_t *img = images + ((int64_t)(hk * gridDim.x + blockIdx.x) * 2 + (blockIdx.z & 1)) * T::KV_BYTES;
  auto row = [&](const float *base, int key) {
    return base + (table ? (((int64_t)table[key / page] * kv_heads + hk) * page + key % page) * D
                         : ((int64_t)hk * max_len + key) * D);
  };
  constexpr int CH = D / 8;
  const int idx = threadIdx.x + (blockIdx.z >> 1) * 256;
  float v[8];
  uint4 t[kTerms];
  uint32_t at;
  if ((blockIdx.z & 1) == 0) {   // 8 columns of a key
    const int r = idx / CH, c = idx % CH;
#pragma unroll
    for (int e = 0; e < 8; ++e)
      v[e] = 0.f;
    if (k0 + r < n_keys) {
      const float4 *p = reinterpret_cast<const float4 *>(row(kc, k0 + r) + 8 * c);
      const float4 a = __ldg(p), b = __ldg(p + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    at = (c >> 3) * (kKeys * 128) + swz(r, c & 7);
  } else {                 // 8 keys of a column; a warp reads 32 columns of a key at once
    const int d = idx % D, c = idx / D;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int key = k0 + 8 * c + e;
      v[e] = key < n_keys ? __ldg(row(vc, key) + d) : 0.f;
    }
    at = swz(d, c);
  }
  split8(v, t);
#pragma unroll
  for (int q = 0; q < kTerms; ++q)
    *reinterpret_cast<uint4 *>(img + q * T::K_PLANE + at) = t[q];
}

struct AttnParams {
  const float *qkv;      // [M][ld]: the q heads come first
  int64_t ld;
  const uint8_t *images; // [kv_heads][key_tiles][K, V]
  int key_tiles;
  float *out;            // [M][ldo]
  int64_t ldo;
  int G, M, pos0, max_len;
  int chunk;             // most key tiles per CTA; a row tile with more is shared by several (gridDim.x at most)
  float *part;           // [kv_heads][row tiles][gridDim.x][kRows * (D + 2)]: unnormalised outputs, then max and sum of the rows
  uint32_t *arrived;     // [kv_heads][row tiles], zeroed by kv_image_kernel
  int *error;
};

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// kind::f16 instruction descriptor: D = f32, A = B = bf16, both K-major, M = 128.
template <int N> __host__ __device__ constexpr uint32_t idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
}
// Executed by a whole warp in uniform control flow (the operands then live in uniform registers), issued by the lane whose
// `leader` is set.
template <int N> __device__ __forceinline__ void mma_ss(uint32_t leader, uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, l;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 l, %5, 0;\n"
      " @l tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc<N>()), "r"(accumulate), "r"(leader)
      : "memory");
}
// A in tensor memory: a row per lane, two bf16 per column
template <int N> __device__ __forceinline__ void mma_ts(uint32_t leader, uint32_t d, uint32_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, l;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 l, %5, 0;\n"
      " @l tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc<N>()), "r"(accumulate), "r"(leader)
      : "memory");
}
// The six products of two three-term numbers: term of A, and place of B's plane in the order of loading (planes 2, 1, 0: a
// plane's slot is free again after 1, 3 and 6 of the products).  The product of the largest terms comes last.
__device__ constexpr int kTermA[6] = {0, 1, 0, 2, 1, 0}, kPlaneOf[6] = {0, 1, 1, 2, 2, 2};
__device__ constexpr bool kFirst[6] = {true, true, false, true, false, false}, kLast[6] = {true, false, true, false, false, true};

template <int D>
__global__ void __launch_bounds__(kThreads, 1) prefill_attn_kernel(const AttnParams p) {
  using T = Tile<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *qs = reinterpret_cast<uint8_t *>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  uint8_t *ks = qs + T::Q_BYTES, *vs = ks + T::K_RING;
  Bars &bars = *reinterpret_cast<Bars *>(vs + T::V_RING);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  volatile int *ab = &bars.abort_flag;
  // the last rows have the longest histories: they start first
  const int qt = gridDim.y - 1 - blockIdx.y, q0 = qt * kRows, hk = blockIdx.z;
  const int last_m = min((q0 + kRows - 1) / p.G, p.M - 1);
  const int n_all = min(p.pos0 + last_m, p.max_len - 1) / kKeys + 1;   // key tiles of the row tile, and this CTA's
  const int splits = (n_all + p.chunk - 1) / p.chunk;
  if ((int)blockIdx.x >= splits)
    return;
  const int t0 = n_all * blockIdx.x / splits, n = n_all * (blockIdx.x + 1) / splits - t0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kKSlots; ++i) {
      mbar_init(&bars.k_full[i], 1);
      mbar_init(&bars.k_empty[i], 1);
    }
    for (int i = 0; i < kTerms; ++i) {
      mbar_init(&bars.v_full[i], 1);
      mbar_init(&bars.v_empty[i], 1);
    }
    mbar_init(&bars.p_ready, kSoftmaxWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars.s_full[i], 1);
      mbar_init(&bars.o_full[i], 1);
    }
    bars.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kSoftmaxWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem_base)), "n"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // ---- Q: three planes of 128 rows, from the rows as they are ---------------------------------------------------------------
  constexpr int CH = D / 8;
#pragma unroll
  for (int i = 0; i < (kRows * CH + kThreads - 1) / kThreads; ++i) {
    const int idx = threadIdx.x + i * kThreads;
    if (idx >= kRows * CH)
      break;
    const int r = idx / CH, c = idx % CH, m = (q0 + r) / p.G, g = q0 + r - m * p.G;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (m < p.M) {
      const float4 *src = reinterpret_cast<const float4 *>(p.qkv + (int64_t)m * p.ld + (int64_t)(hk * p.G + g) * D + 8 * c);
      const float4 a = __ldg(src), b = __ldg(src + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    uint4 t[kTerms];
    split8(v, t);
#pragma unroll
    for (int q = 0; q < kTerms; ++q)
      *reinterpret_cast<uint4 *>(qs + q * T::Q_PLANE + (c >> 3) * (kRows * 128) + swz(r, c & 7)) = t[q];
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars.tmem_base, 0);
  kernel_go();   // not before the allocation: see tensor_core.cuh

  if (warp == kSoftmaxWarps) {
    // ---- loader ----------------------------------------------------------------------------------------------------------------
    if (lane == 0) {
      kernel_wait();
      const uint8_t *img = p.images + ((int64_t)hk * p.key_tiles + t0) * 2 * T::KV_BYTES;
      // plane j of the sequence: tile j / 3, planes 2, 1, 0
      auto load = [&](uint8_t *dst, int j, int z, uint64_t *bar) {
        mbar_expect_tx(bar, T::K_PLANE);
        bulk_load(dst, img + ((int64_t)(j / 3) * 2 + z) * T::KV_BYTES + (2 - j % 3) * T::K_PLANE, T::K_PLANE, bar);
      };
      auto load_k = [&](int j) {
        const int slot = j % kKSlots;
        if (j >= kKSlots && !mbar_wait(&bars.k_empty[slot], (j / kKSlots - 1) & 1, ab, p.error, 711))
          return false;
        load(ks + slot * T::K_PLANE, j, 0, &bars.k_full[slot]);
        return true;
      };
      auto load_v = [&](int j) {
        const int slot = j % kTerms;
        if (j >= kTerms && !mbar_wait(&bars.v_empty[slot], (j / kTerms - 1) & 1, ab, p.error, 712))
          return false;
        load(vs + slot * T::K_PLANE, j, 1, &bars.v_full[slot]);
        return true;
      };
      bool ok = true;
      for (int j = 0; j < min(kKSlots, 3 * n); ++j)
        load_k(j);
      for (int j = 0; j < kTerms; ++j)
        load_v(j);
      // then in the order in which the slots come free: S(0), S(1), PV(0), S(2), PV(1), ..
      for (int t = 0; t < n && ok; ++t) {
        for (int j = kKSlots + 3 * t; j < min(kKSlots + 3 * t + 3, 3 * n) && ok; ++j)
          ok = load_k(j);
        if (t > 0)
          for (int j = 3 * t; j < 3 * t + 3 && ok; ++j)
            ok = load_v(j);
      }
    }
  } else if (warp == kSoftmaxWarps + 1) {
    // ---- tensor core issue -------------------------------------------------------------------------------------------------
    {
      uint32_t leader;
      asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(leader));
      // (offsets are added to the descriptors' 16-byte addresses; unrolled: the issuing thread must keep ahead of 32 clocks)
      const uint64_t dq = smem_desc(smem_u32(qs)), dk = smem_desc(smem_u32(ks)), dv = smem_desc(smem_u32(vs));
      bool ok = true;
      auto scores = [&](int t) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const int j = 3 * t + kPlaneOf[q], slot = j % kKSlots;
          if (kFirst[q]) {
            ok = __all_sync(0xffffffffu, mbar_wait(&bars.k_full[slot], (j / kKSlots) & 1, ab, p.error, 713));
            if (!ok)
              return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          const uint64_t db = dk + ((slot * T::K_PLANE) >> 4);
#pragma unroll
          for (int k = 0; k < D / 16; ++k)
            mma_ss<kKeys>(leader, tmem + kColS + (t & 1) * kKeys,
                          dq + ((kTermA[q] * T::Q_PLANE + (k >> 2) * (kRows * 128) + (k & 3) * 32) >> 4),
                          db + (((k >> 2) * (kKeys * 128) + (k & 3) * 32) >> 4), (q | k) != 0);
          if (kLast[q] && leader)
            tc_commit(&bars.k_empty[slot]);
        }
        if (leader)
          tc_commit(&bars.s_full[t & 1]);
      };
      scores(0);
      for (int t = 0; t < n && ok; ++t) {
        if (t + 1 < n)   // its accumulator was read before P(t - 1) was ready
          scores(t + 1);
        if (ok)
          ok = __all_sync(0xffffffffu, mbar_wait(&bars.p_ready, t & 1, ab, p.error, 715));
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const int slot = kPlaneOf[q];
          if (kFirst[q]) {
            if (ok)
              ok = __all_sync(0xffffffffu, mbar_wait(&bars.v_full[slot], t & 1, ab, p.error, 714));
            if (!ok)
              break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
#pragma unroll
          for (int k = 0; k < kKeys / 16; ++k)
            mma_ts<D>(leader, tmem + kColO + (t & 1) * 128, tmem + kColP + kTermA[q] * (kKeys / 2) + k * 8,
                      dv + ((slot * T::K_PLANE + k * 32) >> 4), (q | k) != 0);
          if (kLast[q] && leader)
            tc_commit(&bars.v_empty[slot]);
        }
        if (ok && leader)
          tc_commit(&bars.o_full[t & 1]);
      }
    }
  } else {
    // ---- softmax -----------------------------------------------------------------------------------------------------------------
    const int quad = warp & 3, half = warp >> 2, r = quad * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
    const float scale = rsqrtf((float)D);
    const int m_row = (q0 + r) / p.G;
    const int qpos = m_row < p.M ? min(p.pos0 + m_row, p.max_len - 1) : -1;
    const int all_from = min(p.pos0 + q0 / p.G, p.max_len - 1);   // keys up to here: every row of the tile
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + quad) : "memory"); };
    float mrow = kSeed, lsum = 0.f, alpha_o = 1.f;   // alpha_o: what the tile whose O comes next did to the max
    float acc[D / 2];
#pragma unroll
    for (int c = 0; c < D / 2; ++c)
      acc[c] = 0.f;
    bool ok = true;
    auto wait = [&](uint64_t *bar, int parity, int code) {   // whole warps leave the poll
      if (ok)
        ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, ab, p.error, code));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    auto add_output = [&](int t) {   // acc = acc * alpha + O(t)
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        uint32_t o[32];
        tmem_load32(lanes + kColO + (t & 1) * 128 + half * (D / 2) + c, o);
        tmem_wait_load();
#pragma unroll
        for (int e = 0; e < 32; ++e)
          acc[c + e] = fmaf(acc[c + e], alpha_o, __uint_as_float(o[e]));
      }
    };
    // (a warp that gave up goes on without waiting: the barriers below keep their count)
    for (int t = 0; t < n; ++t) {
      wait(&bars.s_full[t & 1], (t >> 1) & 1, 716);
      float s[32];
      {
        uint32_t w[32];
        tmem_load32(lanes + kColS + (t & 1) * kKeys + half * 32, w);
        tmem_wait_load();
#pragma unroll
        for (int e = 0; e < 32; ++e)
          s[e] = __uint_as_float(w[e]) * scale;
      }
      const int key0 = (t0 + t) * kKeys + half * 32;
      if ((t0 + t + 1) * kKeys - 1 > all_from) {
#pragma unroll
        for (int e = 0; e < 32; ++e)
          s[e] = key0 + e <= qpos ? s[e] : -INFINITY;   // its exponential is exactly 0
      }
      float mx = s[0];
#pragma unroll
      for (int e = 1; e < 32; ++e)
        mx = fmaxf(mx, s[e]);
      bars.mx[t & 1][half][r] = mx;
      pair_sync();
      const float nm = fmaxf(fmaxf(mrow, mx), bars.mx[t & 1][half ^ 1][r]);
      const float alpha = expf(mrow - nm);
      mrow = nm;
      float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        s[e] = expf(s[e] - nm);
        ps[e & 3] += s[e];
      }
      lsum = fmaf(lsum, alpha, (ps[0] + ps[1]) + (ps[2] + ps[3]));
      if (t > 0)   // also: P is free
        wait(&bars.o_full[(t - 1) & 1], ((t - 1) >> 1) & 1, 717);
#pragma unroll
      for (int q = 0; q < kTerms; ++q) {
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e)
          w[e] = take_bf16(s[2 * e], s[2 * e + 1]);
        tmem_store16(lanes + kColP + q * (kKeys / 2) + half * 16, w);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&bars.p_ready);
      if (t > 0)
        add_output(t - 1);
      alpha_o = alpha;
    }
    wait(&bars.o_full[(n - 1) & 1], ((n - 1) >> 1) & 1, 718);
    add_output(n - 1);
    // ---- the two halves' sums, then whole rows through shared memory (K and V are no longer read) -----------------------------
    bars.sum[half][r] = lsum;
    pair_sync();
    lsum += bars.sum[half ^ 1][r];
    float *stage = reinterpret_cast<float *>(ks);
    const bool whole = splits == 1;
    const float r_sum = __frcp_rn(lsum);
#pragma unroll
    for (int c = 0; c < D / 2; c += 4) {
      float4 o = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      if (whole)
        o = make_float4(quotient(o.x, lsum, r_sum), quotient(o.y, lsum, r_sum), quotient(o.z, lsum, r_sum), quotient(o.w, lsum, r_sum));
      *reinterpret_cast<float4 *>(stage + r * T::LDO + half * (D / 2) + c) = o;
    }
    pair_sync();
    bool mine = ok;
    float *part = p.part + ((int64_t)(hk * gridDim.y + qt) * gridDim.x) * T::PART;
    if (!whole) {   // leave this CTA's share; the last one of the row tile goes on
      kernel_wait();   // the counters are zero
      float *own = part + (int64_t)blockIdx.x * T::PART;
      for (int i = half * 32 + lane; i < 32 * (D / 4); i += 64) {
        const int rr = quad * 32 + i / (D / 4), c = i % (D / 4);
        __stcg(reinterpret_cast<float4 *>(own + rr * D + 4 * c), *reinterpret_cast<const float4 *>(stage + rr * T::LDO + 4 * c));
      }
      if (half == 0)
        __stcg(reinterpret_cast<float2 *>(own + kRows * D) + r, make_float2(mrow, lsum));
      __threadfence();
      asm volatile("bar.sync 5, %0;" ::"n"(kSoftmaxWarps * 32) : "memory");
      if (threadIdx.x == 0)
        bars.last = atomicAdd(p.arrived + hk * gridDim.y + qt, 1u) == (uint32_t)splits - 1;
      asm volatile("bar.sync 5, %0;" ::"n"(kSoftmaxWarps * 32) : "memory");
      __threadfence();
      mine = ok && bars.last;
    }
    // A thread's pieces of the quad's 32 rows: 64 threads, 16 bytes each, 4 at a time
    auto each4 = [&](auto value) {
#pragma unroll 1
      for (int i0 = half * 32 + lane; i0 < 32 * (D / 4); i0 += 4 * 64) {
        float4 o[4];
        value(i0, o);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int rr = quad * 32 + (i0 + 64 * u) / (D / 4), c = (i0 + 64 * u) % (D / 4);
          const int m = (q0 + rr) / p.G, g = q0 + rr - m * p.G;
          if (m < p.M)
            *reinterpret_cast<float4 *>(p.out + (int64_t)m * p.ldo + (int64_t)(hk * p.G + g) * D + 4 * c) = o[u];
        }
      }
    };
    if (mine && whole) {
      each4([&](int i0, float4 (&o)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          o[u] = *reinterpret_cast<const float4 *>(stage + (quad * 32 + (i0 + 64 * u) / (D / 4)) * T::LDO + (i0 + 64 * u) % (D / 4) * 4);
      });
    } else if (mine) {   // rebase the shares on the largest of their maxima; a share's factor per row goes through shared memory
      float *factor = stage;   // [splits][kRows]; the shares have left it
      if (half == 0) {
        float mx = kSeed, l = 0.f;
#pragma unroll 4
        for (int z = 0; z < splits; ++z)
          mx = fmaxf(mx, __ldcg(part + (int64_t)z * T::PART + kRows * D + 2 * r));
#pragma unroll 4
        for (int z = 0; z < splits; ++z) {
          const float2 ml = __ldcg(reinterpret_cast<const float2 *>(part + (int64_t)z * T::PART + kRows * D) + r);
          const float fz = expf(ml.x - mx);
          l = fmaf(ml.y, fz, l);
          factor[z * kRows + r] = fz;
        }
        bars.sum[0][r] = l;
        bars.sum[1][r] = __frcp_rn(l);
      }
      pair_sync();
      each4([&](int i0, float4 (&o)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
        for (int z = 0; z < splits; ++z)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int rr = quad * 32 + (i0 + 64 * u) / (D / 4), c = (i0 + 64 * u) % (D / 4);
            const float4 a = __ldcg(reinterpret_cast<const float4 *>(part + (int64_t)z * T::PART + rr * D) + c);
            const float fz = factor[z * kRows + rr];
            o[u] = make_float4(fmaf(a.x, fz, o[u].x), fmaf(a.y, fz, o[u].y), fmaf(a.z, fz, o[u].z), fmaf(a.w, fz, o[u].w));
          }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int rr = quad * 32 + (i0 + 64 * u) / (D / 4);
          const float l = bars.sum[0][rr], rl = bars.sum[1][rr];
          o[u] = make_float4(quotient(o[u].x, l, rl), quotient(o[u].y, l, rl), quotient(o[u].z, l, rl), quotient(o[u].w, l, rl));
        }
      });
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kSoftmaxWarps + 1) {
    if (*ab) {   // copies and products of an abandoned tile may still be in flight: let them land
      const unsigned long long t0 = now_ns();
      while (now_ns() - t0 < 2000000ull) {
      }
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kCols) : "memory");
  }
}

template <int D>
int launch_attn(const AttnParams &p, const float *kc, const float *vc, int kv_heads, int q_tiles, int max_splits, int n_keys,
                const int32_t *table, int page, uint8_t *images, cudaStream_t st) {
  static RaisedOn raised;
  if (int rc = raise_shared_limit(raised, (const void *)prefill_attn_kernel<D>, Tile<D>::SMEM))
    return rc;
  if (int rc = launch_after(kv_image_kernel<D>, dim3(p.key_tiles, kv_heads, 2 * kKeys * (D / 8) / 256), 256, 0, st, kc, vc,
                            p.max_len, n_keys, table, page, images, p.arrived, max_splits > 1 ? q_tiles * kv_heads : 0))
    return rc;
  return launch_after(prefill_attn_kernel<D>, dim3(max_splits, q_tiles, kv_heads), kThreads, Tile<D>::SMEM, st, p);
}

} // namespace

static int64_t share_bytes(int D) { return (int64_t)kMaxShares * (kRows * (D + 2) + 1) * 4; }

int64_t prefill_attn_workspace_bytes(int n_keys, int kv_heads, int D) {
  return share_bytes(D) + (int64_t)kv_heads * ((n_keys + kKeys - 1) / kKeys) * 2 * kTerms * kKeys * D * 2;
}

bool prefill_attn_takes(const float *qkv, int64_t ld, const float *kc, const float *vc, const float *out, int64_t ldo, int D, int M) {
  return (D == 64 || D == 128) && M >= 64 && (ld & 3) == 0 && (ldo & 3) == 0 &&
         (((uintptr_t)qkv | (uintptr_t)kc | (uintptr_t)vc | (uintptr_t)out) & 15) == 0;
}

int prefill_attn_launch(const float *qkv, int64_t ld, const float *kc, const float *vc, float *out, int64_t ldo, int q_heads,
                        int kv_heads, int D, int max_len, int pos0, int M, const int32_t *table, int page, void *workspace,
                        int64_t workspace_bytes, int *error, cudaStream_t st) {
  const int n_keys = std::min(pos0 + M, max_len);
  if (!workspace || workspace_bytes < prefill_attn_workspace_bytes(n_keys, kv_heads, D))
    return fail(B200_EINVAL, "prefill attention: workspace of %lld bytes is too small", (long long)workspace_bytes);
  AttnParams p{};
  p.qkv = qkv;
  p.ld = ld;
  uint8_t *images = (uint8_t *)workspace + share_bytes(D);
  p.images = images;
  p.part = (float *)workspace;
  p.arrived = (uint32_t *)(p.part + (int64_t)kMaxShares * kRows * (D + 2));
  p.key_tiles = (n_keys + kKeys - 1) / kKeys;
  p.out = out;
  p.ldo = ldo;
  p.G = q_heads / kv_heads;
  p.M = M;
  p.pos0 = pos0;
  p.max_len = max_len;
  p.error = error;
  // Row tiles have histories from pos0 to pos0 + M keys, and few rows make few tiles.  While there are fewer row tiles than
  // SMs their keys are shared out: the smallest shares of which one wave (148 CTAs) holds all, at least 2 key tiles, and none of
  // up to three (a share costs a Q conversion and a trip through L2): 366 rows 3.61 ms a pass with at least 4, 3.54 with 2; 150
  // rows 2.73 whole, 2.82 in two.
  const int q_tiles = (int)(((int64_t)M * p.G + kRows - 1) / kRows), most = p.key_tiles;
  auto shares = [&](int chunk) {
    int64_t n = 0;
    for (int i = 0; i < q_tiles; ++i) {
      const int last = std::min((int)(((int64_t)(i + 1) * kRows - 1) / p.G), M - 1);
      n += (std::min(pos0 + last, max_len - 1) / kKeys + chunk) / chunk;
    }
    return n * kv_heads;
  };
  p.chunk = most;
  auto slots = [&](int chunk) { return (int64_t)((most + chunk - 1) / chunk) * q_tiles * kv_heads; };
  if ((int64_t)q_tiles * kv_heads < kSms) {
    int lo = std::min(most, std::max(most <= 3 ? 3 : 2, (most + kMostSplits - 1) / kMostSplits));
    while (lo < p.chunk) {
      const int mid = (lo + p.chunk) / 2;
      if (shares(mid) <= kSms && slots(mid) <= kMaxShares)
        p.chunk = mid;
      else
        lo = mid + 1;
    }
  }
  const int max_splits = (most + p.chunk - 1) / p.chunk;
  return D == 128 ? launch_attn<128>(p, kc, vc, kv_heads, q_tiles, max_splits, n_keys, table, page, images, st)
                  : launch_attn<64>(p, kc, vc, kv_heads, q_tiles, max_splits, n_keys, table, page, images, st);
}

} // namespace b200
