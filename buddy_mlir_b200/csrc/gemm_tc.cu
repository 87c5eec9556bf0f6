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
// three rows of the A operand: a tile of 128 rows is 42 activation rows x 3 digits (planes; two rows are left over), in the
// k order of the packed weights.  All products and sums are exact integers; the epilogue adds the planes' sums in f32.
// Two bf16 terms per activation and weights converted to bf16, the form before this one, kept 2^-17 of each element; three
// digits keep 2^-23 of the row's largest, which is less where a few channels of a row are far above the rest.  Such rows are
// wide: six digits, in passes of their own over the tile (planes_kernel says which rows, wide_passes what they cost the others).
// Relative error (2-norm, against f64) of the columns that do not use a channel R times the rest, 256 x 1536 x 1536:
//   R            1        30       100      1000     10000
//   now          1.7e-7   1.1e-6   9.4e-7   4.0e-7   8.1e-8
//   three digits 3.2e-7   3.2e-6   1.0e-5   1.1e-4   9.9e-4    (for every row, 23 bits)
//   two bf16     2.5e-6 for all; f32 products and sums 7.0e-7
// Time with no wide row / one / all: 1024 x 17920 x 1536 103 / 112 / 250 us, 1000 x 1536 x 8960 50 / 77 / 139, 24 x 17920 x 1536
// 11.5 / 21 / 29.
// Against bf16: half the bytes of the weight operand and no pass that converts weights; three planes are three times the
// operations of one bf16 product, at 2.4 POP/s (2048 x 8960 x 8960) against 1.6 PFLOP/s.  What few rows need is bytes and
// latency, and what many rows save are the passes around the GEMM.
//
// W8A8 (b200_gemm_w8a8) is the same kernel with one plane: the tile's 128 rows are activation rows.
//
// A CTA computes a 128 x 128 or 128 x 256 tile of sums: warp 0 issues the TMA loads (cp.async.bulk.tensor, no multicast) of
// 128-byte k blocks into a ring of 96 KB (3 stages of 32 KB, or 2 of 48), warp 1 one thread of tcgen05.mma, warps 2..9 the
// epilogue; two CTAs are resident per SM, so one's epilogue runs under the other's main loop.  The weight loads start
// before the activations are there (programmatic dependent launch behind the kernel that makes the planes; chain_start says
// what keeps them behind the caller's earlier work).  The main loop
// is bound by the bytes it brings from L2 (64 bytes per clock and SM), hence 256 columns where that leaves two CTAs
// for every SM (with planes; W8A8 always takes 128, see there).
// Few output tiles: the k range is split over gridDim.z, and the CTA that finishes a tile last adds the shares in order.
//
// Every wait is bounded (poll count and wall time); on expiry the CTA records
// an error, all roles fall through, tensor memory is released and the host
// call fails.
#include "common.cuh"
#include "gemv_mma.cuh"
#include "tensor_core.cuh"

#include <cuda.h>

#include <algorithm>
#include <mutex>

namespace b200 {

namespace {

constexpr int BM = 128;                        // rows of a tile of sums
constexpr int BK = 128;                        // int8 per k block: one 128-byte swizzle row
constexpr int kPlanes = 3, kPlaneRows = 42;    // digits per activation, activation rows per tile
constexpr int kWidePlanes = 6, kWideRows = 21; // the same for rows that need six digits: half a tile's rows at a time
constexpr int kThreads = 320;                  // loader, mma, 8 epilogue warps
constexpr int kEpiWarps = 8;
constexpr int kMaxStages = 3;
constexpr int kSms = 148, kResident = 2 * kSms;   // CTAs of the GEMM that run at once: two per SM
constexpr int kMaxPartialTiles = 320;          // split-K: shares of tiles in the workspace (a little over one per resident CTA)
constexpr int kHeadBytes = 2048;               // workspace head: error word, scales of W8A8, arrival counters

template <int BN> struct Ring {
  static constexpr uint32_t A_BYTES = BM * BK, W_BYTES = BN * BK, STAGE_BYTES = A_BYTES + W_BYTES;
  static constexpr int STAGES = BN == 256 ? 2 : 3;
  static constexpr int SMEM = STAGES * (int)STAGE_BYTES + 1024 + 256;
};

struct Bars {
  uint64_t full[kMaxStages];   // TMA bytes of the stage have landed
  uint64_t empty[kMaxStages];  // the tensor core is done with the stage
  uint64_t accum;              // all MMAs have completed
  uint32_t tmem_base;
  int abort_flag;
  int last;                    // split-K: this CTA completes its tile
  int wide;                    // halves of the tile's rows that have wide rows
};

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap *map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
// kind::i8 instruction descriptor: D = s32, A = B = s8, both K-major, M = 128.
template <int BN>
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
struct GemmParams {
  int M, N, K;                 // K: multiple of 64
  const float *scale, *bias;   // [N], bias may be null
  const float *row_scale;      // planes: [M], negative for wide rows; W8A8: one value
  const float *residual;       // [M, ldr] or null; may alias C
  float *C;                    // [M, ldc]
  int64_t ldc, ldr;
  int silu_pairs;              // columns (2j, 2j+1) are (gate_j, up_j): C[m, j] = silu(g) * u, ldc counts N/2 columns
  int splits;                  // CTAs along K per tile (gridDim.z)
  void *partial;               // [tiles][splits][rows][128]: f32 sums of the planes, or s32 (W8A8)
  uint32_t *arrived;           // [tiles], zeroed by the kernel before
  int *error;
};

// The operations and their order are the reference's.
__device__ __forceinline__ float silu_of(float g, float u) {
  const float sg = 1.0f / (1.0f + expf(-g));   // subgraph0_decode_simplify.mlir:226-231
  return __fmul_rn(__fmul_rn(g, sg), u);
}

// The epilogue warps' part of a pass: a thread reads an accumulator row (its lane of tensor memory) and half of its columns; the
// sums go to a padded tile in shared memory (the ring is idle by then), from where the warps add up the planes and write whole
// rows, warp w rows w, w + 8, .. of the pass: lane j holds the scale of the j-th of them (row_scales).  SIX: the pass over the wide
// rows of one half of the tile's rows.
template <bool PLANES> __device__ __forceinline__ float row_scales(const GemmParams &p, int first, int rows) {
  if (!PLANES)
    return p.row_scale[0];
  const int r = ((int)threadIdx.x >> 5) - 2 + (threadIdx.x & 31) * kEpiWarps;
  return r < rows ? p.row_scale[blockIdx.y * kPlaneRows + first + r] : 0.f;
}
template <int BN, bool PLANES, bool SIX>
__device__ __forceinline__ void store_tile(const GemmParams &p, Bars &bars, uint8_t *tiles, uint32_t tmem, bool ok, int half,
                                           float scales) {
  constexpr int kRows = PLANES ? kPlaneRows : BM;   // activation rows of the tile
  constexpr int kStep = SIX ? kWideRows : kRows;
  constexpr int kFold = SIX ? 1 : 8;                // shares of a split tile in flight
  constexpr int LDS = 128 + 4;                      // row stride of the staging tile, in words
  float *ep = reinterpret_cast<float *>(tiles);     // [BM][LDS]: 66 KB of the ring
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ew = warp - 2, quad = warp & 3;
  const int m0 = blockIdx.y * kRows, n0 = blockIdx.x * BN, rows_all = min(kRows, p.M - m0);
  const int first = SIX ? half * kWideRows : 0, rows = min(kStep, rows_all - first);   // the pass's rows of the tile
#pragma unroll 1
  for (int h = 0; h < BN / 128; ++h) {   // 128 columns of the accumulator at a time
    const int nh = n0 + h * 128;
    if (nh >= p.N)
      break;
    if (h > 0)   // the staging tile is free again once the previous half has been stored
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
    if (ok && (PLANES || quad * 32 < p.M - m0)) {   // lanes beyond M hold nothing
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // a warp reads the 32 lanes of tensor memory that match its rank within its warpgroup; the two warps that share a
      // lane quarter take half the columns each
      const int row = quad * 32 + lane, cb0 = (ew >> 2) * 64;
      const int d = row / kStep;   // PLANES: which digit; its weight is 2^16, 2^8, 1, 2^-7, 2^-15, 2^-23
      const float f = __uint_as_float((uint32_t)(127 + 16 - 8 * d + (d >= kPlanes)) << 23);
#pragma unroll 1
      for (int cb = cb0; cb < cb0 + 64; cb += 32) {
        uint32_t v[32];
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(h * 128 + cb);
        tmem_load32(taddr, v);
        tmem_wait_load();
        float *erow = ep + row * LDS + cb;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          float4 o;
          if (PLANES)
            o = make_float4(__int2float_rn((int)v[j]) * f, __int2float_rn((int)v[j + 1]) * f,
                            __int2float_rn((int)v[j + 2]) * f, __int2float_rn((int)v[j + 3]) * f);
          else
            o = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]),
                            __uint_as_float(v[j + 3]));
          *reinterpret_cast<float4 *>(erow + j) = o;
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
    const int cols = min(128, p.N - nh);
    // sums of the pass's row r, columns c .. c + 3 of this CTA's k range
    auto sums = [&](int r, int c) {
      float4 a = *reinterpret_cast<const float4 *>(ep + r * LDS + c);
      if (PLANES) {
#pragma unroll
        for (int q = 1; q < (SIX ? kWidePlanes : kPlanes); ++q) {
          const float4 b = *reinterpret_cast<const float4 *>(ep + (q * kStep + r) * LDS + c);
          a = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
        }
      }
      return a;
    };
    bool mine = ok;
    int r0 = first, nr = rows;   // the rows to finish
    const int tile = blockIdx.y * gridDim.x + blockIdx.x;
    float4 *shares = reinterpret_cast<float4 *>(p.partial) + (int64_t)tile * p.splits * kRows * 32;
    if (p.splits > 1) {   // (BN = 128) leave this CTA's share; after its last pass the last CTA of the tile goes on
      if (ok)   // (a wide row's share is written again by the pass with six digits, which has nothing for other rows)
#pragma unroll 1
        for (int r = ew, j = 0; r < rows; r += kEpiWarps, ++j)
          if (!SIX || signbit(__shfl_sync(0xffffffffu, scales, j)))
            __stcg(shares + ((int64_t)blockIdx.z * kRows + first + r) * 32 + lane, sums(r, lane * 4));
      mine = false;
      if (!PLANES || bars.wide >> (SIX ? half + 1 : 0) == 0) {
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        if (threadIdx.x == 64)
          bars.last = atomicAdd(p.arrived + tile, 1u) == (uint32_t)p.splits - 1;
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        __threadfence();
        mine = ok && bars.last;
      }
      r0 = 0;
      nr = rows_all;
      if (SIX)
        scales = row_scales<PLANES>(p, 0, rows_all);
    }
    if (mine) {
      const bool vec = (p.ldc & 3) == 0 && ((uintptr_t)p.C & 15) == 0 && (p.N & 3) == 0 &&
                       (!p.residual || ((p.ldr & 3) == 0 && ((uintptr_t)p.residual & 15) == 0));
#pragma unroll 1
      for (int r = ew, j = 0; r < nr; r += kEpiWarps, ++j) {
        const float rs = PLANES ? __shfl_sync(0xffffffffu, scales, j) : scales;
        const int i = r * 32 + lane, c = lane * 4, m = m0 + r0 + r, n = nh + c;
        if (c >= cols || (PLANES && p.splits == 1 && signbit(rs) != SIX))   // (finished by another pass)
          continue;
        float y[4];
        if (p.splits > 1) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int z0 = 0; z0 < p.splits; z0 += kFold) {
            float4 b[kFold];
#pragma unroll
            for (int z = 0; z < kFold; ++z)
              b[z] = z0 + z < p.splits ? __ldcg(shares + (int64_t)(z0 + z) * kRows * 32 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int z = 0; z < kFold; ++z)
              if (PLANES)
                a = make_float4(a.x + b[z].x, a.y + b[z].y, a.z + b[z].z, a.w + b[z].w);
              else
                a = make_float4(__int_as_float(__float_as_int(a.x) + __float_as_int(b[z].x)),
                                __int_as_float(__float_as_int(a.y) + __float_as_int(b[z].y)),
                                __int_as_float(__float_as_int(a.z) + __float_as_int(b[z].z)),
                                __int_as_float(__float_as_int(a.w) + __float_as_int(b[z].w)));
          }
          y[0] = a.x; y[1] = a.y; y[2] = a.z; y[3] = a.w;
        } else {
          const float4 a = sums(r, c);
          y[0] = a.x; y[1] = a.y; y[2] = a.z; y[3] = a.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int ne = min(n + e, p.N - 1);
          if (PLANES)
            y[e] = __fmul_rn(__fmul_rn(y[e], fabsf(rs)), __ldg(p.scale + ne));
          else   // linalg.py:12836-12846: float(acc) * (act_scale * weight_scale[n])
            y[e] = __fmul_rn(__int2float_rn(__float_as_int(y[e])), __fmul_rn(rs, __ldg(p.scale + ne)));
          if (p.bias)
            y[e] = __fadd_rn(y[e], __ldg(p.bias + ne));
        }
        if (p.silu_pairs) {
          float *dst = p.C + (int64_t)m * p.ldc + (n >> 1);
          dst[0] = silu_of(y[0], y[1]);
          if (n + 3 < p.N)   // N is even
            dst[1] = silu_of(y[2], y[3]);
        } else {
          float *dst = p.C + (int64_t)m * p.ldc + n;
          const float *res = p.residual + (int64_t)m * p.ldr + n;
          if (vec) {
            if (p.residual) {
              const float4 q = *reinterpret_cast<const float4 *>(res);
              y[0] = __fadd_rn(q.x, y[0]);
              y[1] = __fadd_rn(q.y, y[1]);
              y[2] = __fadd_rn(q.z, y[2]);
              y[3] = __fadd_rn(q.w, y[3]);
            }
            *reinterpret_cast<float4 *>(dst) = make_float4(y[0], y[1], y[2], y[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n + e < p.N)
                dst[e] = p.residual ? __fadd_rn(res[e], y[e]) : y[e];
          }
        }
      }
    }
  }
}

// The tile's wide rows once more, with six digits: a half of its rows at a time (`halves`: which).  Everything a normal tile does
// again, in a function of its own and with little code, since code counts even where it does not run: without wide rows,
// 24 x 17920 x 1536 takes 13.5 us without this function, 13.9 with it, 16.3 with its loops unrolled as a tile's were;
// 1024 x 17920 x 1536 106.8, 108.4, and 110.5 with these passes as a loop around the tile's code.  For the same reason the loops
// over the rows of a tile are not unrolled (prefill of 1000 rows: 7.59 -> 7.48 ms).
template <int BN>
__device__ __noinline__ void wide_passes(const CUtensorMap &map_x, const CUtensorMap &map_w, const GemmParams &p) {
  using R = Ring<BN>;
  constexpr int S = R::STAGES;
  extern __shared__ __align__(1024) uint8_t smem[];   // (all found again, so that the caller keeps nothing for it)
  uint8_t *tiles = reinterpret_cast<uint8_t *>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  Bars &bars = *reinterpret_cast<Bars *>(tiles + S * R::STAGE_BYTES);
  const uint32_t tmem = bars.tmem_base;
  const int nkb_all = (p.K + BK - 1) / BK;
  const int kb0 = nkb_all * blockIdx.z / p.splits, nkb = nkb_all * (blockIdx.z + 1) / p.splits - kb0;
  volatile int *ab = &bars.abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, halves = bars.wide;
  int g = nkb, phase = 1;   // k blocks that have gone through the ring, parity of the accumulator's barrier
  for (int half = 0; half < 2; ++half) {
    if (!(halves >> half & 1))
      continue;
    if (warp == 0) {
      if (lane == 0)
        for (int i = 0; i < nkb; ++i) {
          const int s = (g + i) % S, u = (g + i) / S;
          if (u > 0 && !mbar_wait(&bars.empty[s], (u - 1) & 1, ab, p.error, 701))
            break;
          mbar_expect_tx(&bars.full[s], R::STAGE_BYTES);
          tma_load_2d(tiles + s * R::STAGE_BYTES + R::A_BYTES, &map_w, (kb0 + i) * BK, blockIdx.x * BN, &bars.full[s]);
          tma_load_2d(tiles + s * R::STAGE_BYTES, &map_x, (kb0 + i) * BK, (blockIdx.y * 2 + half) * BM, &bars.full[s]);
        }
    } else if (warp == 1) {
      if (lane == 0) {
        for (int i = 0; i < nkb; ++i) {
          const int s = (g + i) % S;
          if (!mbar_wait(&bars.full[s], ((g + i) / S) & 1, ab, p.error, 702))
            break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = smem_u32(tiles + s * R::STAGE_BYTES), w = a + R::A_BYTES;
#pragma unroll 1
          for (int k = 0; k < BK / 32; ++k)
            mma_i8<BN>(tmem, smem_desc(a + k * 32), smem_desc(w + k * 32), (i | k) != 0);
          tc_commit(&bars.empty[s]);
        }
        tc_commit(&bars.accum);
      }
    } else {
      const int first = half * kWideRows;
      const float scales = row_scales<true>(p, first, min(kWideRows, p.M - (int)blockIdx.y * kPlaneRows - first));
      const bool ok = mbar_wait(&bars.accum, phase, ab, p.error, 703) && !*ab;
      store_tile<BN, true, true>(p, bars, tiles, tmem, ok, half, scales);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the next pass loads over the staging tile
    }
    g += nkb;
    phase ^= 1;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (*ab)
      break;
  }
}

// SLIM: 64 registers a thread, so that a CTA of this GEMM, one of the kernel that makes the digits and one of the next GEMM,
// which loads its weights meanwhile, are on an SM at once.  A decode step of 6 / 12 / 16 / 20 sequences takes 2.23 / 2.31 / 2.38 /
// 2.50 ms with it and 2.39 / 2.47 / 2.49 / 2.61 without; at 24 rows it depends on the contexts, 32 and 42 rows take 2.89 / 3.00
// with it and 2.83 / 2.93 without.
template <int BN, bool PLANES, bool SLIM>
__global__ void __launch_bounds__(kThreads, SLIM ? 3 : 2)
gemm_i8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_x) {
  using R = Ring<BN>;
  constexpr int S = R::STAGES;
  constexpr int kRows = PLANES ? kPlaneRows : BM;   // activation rows of the tile
  extern __shared__ __align__(1024) uint8_t smem[];
  // 1024-byte alignment of every swizzled tile
  uint8_t *tiles = reinterpret_cast<uint8_t *>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  Bars &bars = *reinterpret_cast<Bars *>(tiles + S * R::STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kRows, n0 = blockIdx.x * BN;
  // this CTA's share of the k blocks
  const int nkb_all = (p.K + BK - 1) / BK;
  const int kb0 = nkb_all * blockIdx.z / p.splits, nkb = nkb_all * (blockIdx.z + 1) / p.splits - kb0;
  volatile int *ab = &bars.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    mbar_init(&bars.accum, 1);
    bars.abort_flag = 0;
    bars.wide = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {   // tensor memory: one warp allocates, the same warp frees
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem_base)), "n"(BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = bars.tmem_base;
  kernel_go();   // not before the allocation: see tensor_core.cuh

  if (warp == 0) {
    // ---- loader --------------------------------------------------------------------------------------------------
    if (lane == 0) {
      auto load_w = [&](int i) {
        const int s = i % S;
        mbar_expect_tx(&bars.full[s], R::STAGE_BYTES);
        tma_load_2d(tiles + s * R::STAGE_BYTES + R::A_BYTES, &map_w, (kb0 + i) * BK, n0, &bars.full[s]);
      };
      auto load_a = [&](int i) {
        const int s = i % S;
        tma_load_2d(tiles + s * R::STAGE_BYTES, &map_a, (kb0 + i) * BK, blockIdx.y * BM, &bars.full[s]);
      };
      // few rows: the weights' way from memory is the GEMM; all of this CTA's share starts for L2 while the kernels before run
      // (if all CTAs are resident at once: 24 x 151936 x 1536, 594 CTAs, took 68 us with it and 60 without)
      if (gridDim.y <= 2 && gridDim.x * gridDim.y * gridDim.z <= kResident)
        for (int i = S; i < nkb; ++i)
          tma_prefetch_2d(&map_w, (kb0 + i) * BK, n0);
      const int ahead = min(S, nkb);
      for (int i = 0; i < ahead; ++i)   // the weights do not wait for the kernel before
        load_w(i);
      kernel_wait();
      for (int i = 0; i < ahead; ++i)
        load_a(i);
      for (int i = ahead; i < nkb; ++i) {
        if (!mbar_wait(&bars.empty[i % S], (i / S - 1) & 1, ab, p.error, 701))
          break;
        load_w(i);
        load_a(i);
      }
    }
  } else if (warp == 1) {
    // ---- tensor core issue (one thread) -----------------------------------------------------------------------------
    if (lane == 0) {
      for (int i = 0; i < nkb; ++i) {
        const int s = i % S;
        if (!mbar_wait(&bars.full[s], (i / S) & 1, ab, p.error, 702))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = smem_u32(tiles + s * R::STAGE_BYTES), w = a + R::A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / 32; ++k)   // 32 int8 = 32 bytes along the swizzled row
          mma_i8<BN>(tmem, smem_desc(a + k * 32), smem_desc(w + k * 32), (i | k) != 0);
        tc_commit(&bars.empty[s]);   // arrives when the MMAs above have read the stage
      }
      tc_commit(&bars.accum);
    }
  } else {
    // ---- epilogue ----------------------------------------------------------------------------------------------------
    kernel_wait();   // row scales, counters
    const float scales = row_scales<PLANES>(p, 0, min(kRows, p.M - m0));
    if (PLANES) {
      const uint32_t wide = __ballot_sync(0xffffffffu, signbit(scales));
      if (wide != 0 && lane == 0)   // rows warp - 2 + 8 j, the first half of the tile: below 21
        for (int j = 0; j < (kRows + kEpiWarps - 1) / kEpiWarps; ++j)
          if (wide >> j & 1)
            atomicOr(&bars.wide, warp - 2 + kEpiWarps * j < kWideRows ? 1 : 2);
    }
    const bool ok = mbar_wait(&bars.accum, 0, ab, p.error, 703) && !*ab;
    store_tile<BN, PLANES, false>(p, bars, tiles, tmem, ok, 0, scales);
    if (PLANES)
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // a pass over wide rows loads over the staging tile
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PLANES && bars.wide != 0 && !*ab) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    wide_passes<BN>(map_x, map_w, p);
  }
  if (warp == 1) {
    if (*ab) {   // copies of an abandoned tile may still be in flight: let them land before the CTA ends
      const unsigned long long t0 = now_ns();
      while (now_ns() - t0 < 2000000ull) {
      }
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(BN) : "memory");
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

// A[M,K] f32 -> planes [ceil(M/42)][3][42] (+ 2 unused rows) [K] int8 in the k order of the packed weight rows, and the rows'
// scales (the sign says that a row is wide); optional RMSNorm of every row (the factor 1/rms goes into the scale).  T threads per row, a thread takes 16-byte
// units: it reads four groups of four k and writes whole 16-byte pieces of the planes.  The row is read once and stays in
// registers up to 48 T elements.  Also clears the GEMM's counters and, outside a pass, its error word (head).
//
// Wide rows.  Rounding to a unit leaves 0.29 units (rms) in every element, which must be no more than the 2^-19 of an element
// that two bf16 terms leave: the row's bulk has to have an rms of at least 2^17 units.  Its bulk is what lies below a quarter of
// the largest magnitude, and is also to have a mean of 2^16, so that a few percent of large elements do not pass for bulk.  A
// row with channels more than about 32 times the rest misses that, and is written a second time, into `wides`
// [ceil(M/42)][2][6][21] (+ 2 rows) [K]: three more digits, of what the first three leave over in units of 2^-23, exact down to
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
  uint8_t *dst = planes + ((int64_t)(m / kPlaneRows) * BM + m % kPlaneRows) * K;
  uint8_t *wdst = wides + ((int64_t)(m / kWideRows) * BM + m % kWideRows) * K;   // (42 = 2 x 21)
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
          *reinterpret_cast<uint4 *>(dst + (int64_t)pl * kPlaneRows * K + u * 16) =
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
      uint4 *at = reinterpret_cast<uint4 *>(wdst + (int64_t)pl * kWideRows * K + u * 16);
      *at = make_uint4(w[0][pl + 1], w[1][pl + 1], w[2][pl + 1], w[3][pl + 1]);
      *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(at) + (int64_t)kPlanes * kWideRows * K) =
          make_uint4(l[0][pl + 1], l[1][pl + 1], l[2][pl + 1], l[3][pl + 1]);
    }
  }
}

// ---- W8A8: one dynamic scale for the whole activation tensor -------------------------------------------------------------
// buddy-mlir's QuantizedMatmulOp (frontend/Python/ops/linalg.py:12728-12846): s = max(absmax / 127, 1e-10),
// q = clamp(rne(x * (1 / s)), -128, 127), an exact i8 x i8 -> i32 contraction, y = float(acc) * (s * weight_scale[n])
// (+ bias).  Every step is reproduced operation by operation, so the result is bit-identical to the reference arithmetic.
constexpr int kMaxParts = 256;   // partial maxima, in the workspace head

// max |x| of every CTA's share of the tensor (non-negative floats order like their bit patterns); clears the GEMM's counters
// and its error word (null in a pass: the word collects what any of its GEMMs leaves).
__global__ void __launch_bounds__(256)
absmax_kernel(const float *A, int64_t lda, int M, int K, int vec, uint32_t *part, uint32_t *error, uint32_t *arrived,
              int in_pass) {
  chain_start(in_pass);
  __shared__ uint32_t s_mx[8];
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0 && error != nullptr)
      *error = 0u;
    for (int i = threadIdx.x; i < kMaxPartialTiles; i += 256)
      arrived[i] = 0u;
  }
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

template <int BN, bool PLANES, bool SLIM = false>
int launch_gemm(const void *a, int a_rows, const void *x, const void *w, GemmParams &p, int m_tiles, cudaStream_t st) {
  CUtensorMap map_a, map_w, map_x;
  if (int rc = make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, BK, const_cast<void *>(a), p.K, a_rows, (uint64_t)p.K,
                        CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, BK, const_cast<void *>(w), p.K, p.N, (uint64_t)p.K,
                        CU_TENSOR_MAP_SWIZZLE_128B, BN))
    return rc;
  map_x = map_a;
  if (PLANES)
    if (int rc = make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, BK, const_cast<void *>(x), p.K, 2 * (uint64_t)a_rows,
                          (uint64_t)p.K, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  static RaisedOn raised;
  if (int rc = raise_shared_limit(raised, (const void *)gemm_i8_kernel<BN, PLANES, SLIM>, Ring<BN>::SMEM))
    return rc;
  return launch_after(gemm_i8_kernel<BN, PLANES, SLIM>, dim3((p.N + BN - 1) / BN, m_tiles, p.splits), kThreads, Ring<BN>::SMEM, st,
                      map_a, map_w, p, map_x);
}

// CTAs along K for `tiles` output tiles of `nkb` k blocks: up to two CTAs per SM, within the workspace, at least 8 k
// blocks each: a share's trip through L2 costs what 8 to 12 blocks cost.  24 x 2048 x 1536 (12 blocks): 10.1 us whole, 11.1 in
// 6 shares; 24 x 1536 x 8960 (70 blocks): 27 us whole, 14.4 in 8, 17.2 in 24; 366 x 1536 x 8960 (108 tiles): 34.8 whole, 28.2 in 2.
// A row of a tile's sums costs as much on that trip as 0.4 blocks, so tiles with many rows split only long k ranges (W8A8,
// 1024 x 1536 x 8960: 49.8 us whole, 55.3 in 3; 200 x 4096 x 4096: 21.4 whole, 29 in 4; 64 x 1536 x 8960: 32.2 whole, 19.7 in 8).
int split_k(int tiles, int nkb, int rows) {
  if (tiles >= kSms)
    return 1;
  const int s = std::max(1, std::min({kResident / tiles, nkb / 8, kMaxPartialTiles / tiles}));
  return (nkb - nkb / s) * 5 > rows * 2 ? s : 1;
}

} // namespace

} // namespace b200

using namespace b200;

extern "C" {

int64_t b200_gemm_w8_workspace_bytes(int M, int64_t K) {
  if (M < 1 || K < 1)
    return 0;
  const int64_t tiles = (M + kPlaneRows - 1) / kPlaneRows, Kp = packed_k(B200_W_I8, K);
  // head, row scales, planes, the wide rows' planes, the shares of split tiles
  return kHeadBytes + tiles * kPlaneRows * 4 + 255 + 3 * tiles * BM * Kp + (int64_t)kMaxPartialTiles * kPlaneRows * 128 * 4;
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
  const int K = (int)w->K, N = (int)w->N, m_tiles = (M + kPlaneRows - 1) / kPlaneRows;
  char *ws = (char *)workspace;
  float *row_scale = reinterpret_cast<float *>(ws + kHeadBytes);
  uint8_t *planes = reinterpret_cast<uint8_t *>(ws + (kHeadBytes + (int64_t)m_tiles * kPlaneRows * 4 + 255) / 256 * 256);
  uint8_t *wides = planes + (int64_t)m_tiles * BM * K;
  GemmParams p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.scale = (const float *)w->scale;
  p.bias = (const float *)w->bias;
  p.row_scale = row_scale;
  p.residual = residual;
  p.C = C;
  p.ldc = ldc;
  p.ldr = ldr;
  p.silu_pairs = silu_pairs;
  p.partial = wides + (int64_t)m_tiles * 2 * BM * K;
  p.error = reinterpret_cast<int *>(ws);
  p.arrived = reinterpret_cast<uint32_t *>(ws) + 16;
  // threads per row: as few as keep it in registers, more when there are few rows
  int T = 32;
  while (T < 256 && (K > T * 16 * kUnits || (int64_t)M * T < kSms * 256))
    T *= 2;
  const int vec = (lda & 3) == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)norm_weight & 15) == 0;
  if (int rc = launch_after(planes_kernel, dim3((M + 256 / T - 1) / (256 / T)), 256, 0, st, A, lda, M, K, norm_weight, norm_eps, T,
                            vec, planes, row_scale, in_pass ? p.arrived : reinterpret_cast<uint32_t *>(ws),
                            in_pass ? kMaxPartialTiles : 16 + kMaxPartialTiles, in_pass ? 1 : 0, wides))
    return rc;
  // 256 columns per CTA (fewer bytes per operation) when that still gives every SM its two CTAs
  if ((int64_t)((N + 255) / 256) * m_tiles >= kResident) {
    p.splits = 1;
    return launch_gemm<256, true>(planes, m_tiles * BM, wides, w->w, p, m_tiles, st);
  }
  p.splits = split_k((N + 127) / 128 * m_tiles, (K + BK - 1) / BK, std::min(M, kPlaneRows));
  if (M <= 20)
    return launch_gemm<128, true, true>(planes, m_tiles * BM, wides, w->w, p, m_tiles, st);
  return launch_gemm<128, true>(planes, m_tiles * BM, wides, w->w, p, m_tiles, st);
}
} // namespace b200

extern "C" {

/* W8A8 (buddy-mlir's QuantizedMatmulOp): workspace = b200_gemm_w8a8_workspace_bytes(M, K). */
int64_t b200_gemm_w8a8_workspace_bytes(int M, int64_t K) {
  if (M < 1 || K < 1)
    return 0;
  return kHeadBytes + kMaxParts * 4 + ((int64_t)M * K + 255) / 256 * 256 + (int64_t)kMaxPartialTiles * BM * 128 * 4;
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
  const int K = (int)w->K, N = (int)w->N, m_tiles = (M + BM - 1) / BM;
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
  p.partial = q + ((int64_t)M * K + 255) / 256 * 256;
  p.error = reinterpret_cast<int *>(ws);
  p.arrived = reinterpret_cast<uint32_t *>(ws) + 16;
  const int vec = (lda & 3) == 0 && ((uintptr_t)A & 15) == 0;
  const int parts = (int)std::min<int64_t>(((int64_t)M * K / 4 + 1023) / 1024, kMaxParts);
  if (int rc = launch_after(absmax_kernel, dim3(parts), 256, 0, st, A, lda, M, K, vec, part,
                            in_pass ? nullptr : reinterpret_cast<uint32_t *>(ws), p.arrived, in_pass ? 1 : 0))
    return rc;
  const int64_t units = (int64_t)M * (K / 16);
  if (int rc = launch_after(quantize_kernel, dim3((unsigned)((units + 255) / 256)), 256, 0, st, A, lda, M, K, vec,
                            (const uint32_t *)part, parts, act_scale, q))
    return rc;
  // 128 columns for all: with 256, where that leaves two CTAs for every SM, 2048 x 20000 x 8960 takes 423 us instead of 482 and
  // 2048 x 17920 x 1536 105 instead of 112, but 1024 x 18992 x 1536 73 instead of 69 and 600 x 17920 x 1536 51 instead of 47
  p.splits = split_k((N + 127) / 128 * m_tiles, (K + BK - 1) / BK, std::min(M, BM));
  return launch_gemm<128, false>(q, M, q, w->w, p, m_tiles, st);
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
