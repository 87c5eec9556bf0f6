// One persistent kernel per decode token (batch 1): int8, int4 (group 128 or per channel) and f32 weights.
//
// What bounds a decode step is not bytes alone: a layer is a chain of small dependent projections, and every one of
// them pays its start-up (launch, instruction fetch, first loads) and the hand-over of its result.  One CTA per SM
// therefore stays resident for the whole token:
//
//  * Weights.  Every WARP owns a private stream: the 2 KB blocks (16 rows of a tile x some k, already in the order the
//    lanes read them) it will consume during the token, back to back, over all layers and projections.  A small ring per
//    warp is filled with cp.async, every lane copying exactly the 16-byte pieces it will read itself: no producer, no
//    barrier, and refills never wait for activations, so the memory system stays busy across the dependency points of the
//    graph.  (Bulk copies of the same blocks: issuing one holds the warp for about 400 clocks, more than its math.)
//  * Activations.  There is no grid-wide barrier.  Every vector that crosses CTAs is stored as 8-byte (value, tag)
//    pairs; the tag names launch, layer and producer.  A consumer polls the pairs it needs: arrival IS the
//    synchronisation.  Buffers alternate by layer parity; a value is only overwritten two layers later, which needs
//    every CTA's output of the layer in between, so nobody can still be reading it.
//  * Math.  int8 and int4 rows go through the integer tensor cores with the activations as four int8 planes
//    (gemv_mma.cuh: exact sums, no dequantisation); f32 rows through FFMA.
//  * Code.  One body serves all projections, as loops, and the whole layer is kept small: a phase is a microsecond long, and
//    what does not stay in the instruction cache (about 100 KB; then 22 clocks per instruction) is paid for in every one.
//
// Every wait (mbarrier or tag poll) is bounded: on expiry the kernel records an error code, all later waits fall
// through, control flow stays identical (so CTA barriers stay matched), and the host call fails.
//
// Arithmetic is that of examples/BuddyDeepSeekR1/subgraph0_decode_simplify.mlir:46-260 with the dequantising GEMVs of
// midend/lib/Conversion/MatMulOptimization/DequantMatMulVectorizationDecode.cpp:250-321 and
// Int4DequantMatMulVectorizationDecode.cpp:359-430, and the attention recurrence of
// frontend/Python/ops/tosa.py:14245-14594.
#include "decode.cuh"
#include "quotient.cuh"
#include "gemv_mma.cuh"

#include <algorithm>
#include <cstddef>

namespace b200 {

namespace {

constexpr int kCT = kDecThreads;
constexpr uint32_t kSpinLimit = 1u << 26;              // poll count bound, and
constexpr unsigned long long kWaitNs = 1000000000ull;  // wall-time bound (1 s) of any single wait
constexpr float kSeed = -1.0e30f;
constexpr int D = 128;                                 // head_dim (checked on the host)
constexpr int kXBatch = 3;                             // groups of four activations a thread has in flight
constexpr int kSet = kSetBytes<4>;                     // planes of 64 k
constexpr int kMaxTiles = 128;                         // tiles of one projection per CTA

// producer phases that tag their outputs
enum { T_QKV = 1, T_ATTN = 2, T_XB = 3, T_MID = 4, T_XA = 5, T_PART = 6, T_CAND = 7 };

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// a / b for a normal b of up to 2^125: the hardware's approximate reciprocal, improved by a step of Newton's iteration, and a product.
// Within an ulp and a half.
__device__ __forceinline__ float div_normal(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return a * newton_reciprocal(b, r);
}
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ll_store(uint2 *p, float v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(tag) : "memory");
}
__device__ __forceinline__ uint2 ll_load1(const uint2 *p) {
  uint2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ll_load2(const uint2 *p) {   // two pairs, 16-byte aligned
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// Bring [p, p + bytes) to L2 (whole 16-byte pieces; p 16-byte aligned).  One thread.
__device__ __forceinline__ void prefetch_l2(const void *p, int64_t bytes) {
  const uint32_t n = (uint32_t)bytes & ~15u;
  if (n > 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(n) : "memory");
}

struct Shared {
  DecParams p;                  // a copy for the function that cannot reach the kernel's parameters cheaply
  alignas(16) float redf[kDecWarps];     // per-warp sum of squares
  float bestv[kDecWarps];
  int besti[kDecWarps];
  float cs[D / 2], sn[D / 2];   // cos / sin of this step's position
  int tile0[5], tiles[5];       // this CTA's tiles of every projection
  int first[5][kDecWarps + 1];  // first block of every warp, in this CTA's list of blocks (tile by tile)
  int ftile[5][kDecWarps];      // and its tile
  int abort_flag;
  // attention: this CTA's (kv head, key range), or head -1; the number of key ranges; its outputs of the fold (in fours)
  int a_head, a_split, a_first, a_end, splits, out0, out1;
  uint8_t wfirst[5][kMaxTiles], wlast[5][kMaxTiles];   // warps that hold shares of a tile
};

static_assert(offsetof(Shared, redf) % 16 == 0, "read as float4");

struct Ctx {
  const DecParams &p;
  Shared &sh;
  const DecLayer *layers;   // shared-memory copy
  uint8_t *planes;          // activation planes or values; attention scratch
  float *part;              // partial sums of the tiles, [part_rows][16]
  uint32_t ring;            // this warp's ring (shared-memory address)
  const uint8_t *ring_ptr;
  const uint8_t *src;       // this warp's stream: next block to request (+ the lane's piece of it)
  int left;                 // blocks not requested yet
  int slot;                 // ring slot that is consumed and refilled next
  uint64_t policy;          // the weights pass through L2 once: caches, scales and norms stay
  int tid, lane, warp;
  uint32_t tag_base;
  long long *tr;            // this CTA's trace rows, or null
};

__device__ __forceinline__ uint32_t tag_of(const Ctx &c, int layer, int what) {
  return c.tag_base + (uint32_t)((layer + 1) * 8 + what);
}
__device__ __forceinline__ void trace(Ctx &c, int layer, int at) {
  if (c.tr != nullptr && c.tid == 0)
    c.tr[layer * kDecTraceSlots + at] = clock64();
}

// Every 1024th step of a poll loop: 0 = give up (recorded), else the time the wait began.
__device__ __noinline__ unsigned long long poll_slow(int *error, volatile int *abort_flag, uint32_t it, unsigned long long t0,
                                                     int code) {
  const unsigned long long t = now_ns();
  if (t0 == 0)
    t0 = t;
  if (*(volatile int *)error == 0 && t - t0 <= kWaitNs && it < kSpinLimit)
    return t0;
  atomicCAS(error, 0, code);
  *abort_flag = 1;
  return 0;
}
struct Poll {
  uint32_t it = 0;
  unsigned long long t0 = 0;
};
__device__ __forceinline__ bool poll_expired(const DecParams &p, Shared &sh, Poll &w, int code) {
  volatile int *ab = &sh.abort_flag;
  if (*ab)
    return true;
  if ((++w.it & 0x3FF) == 0) {
    w.t0 = poll_slow(p.error, ab, w.it, w.t0, code);
    return w.t0 == 0;
  }
  return false;
}
// The same for a whole warp, lanes with `ok` still waiting for the others: one decision for all of them.  Poll loops leave
// together: lanes that fall out of a loop one by one stay apart, and every shuffle after it pays for it.  (No sleep between polls:
// with 20 ns a 1.5B int8 step at contexts 97 / 1000 takes 643 / 668 us instead of 640 / 664.)
__device__ __forceinline__ bool poll_done(const DecParams &p, Shared &sh, Poll &w, int code, bool ok) {
  if (__all_sync(0xffffffffu, ok))
    return true;
  return __any_sync(0xffffffffu, poll_expired(p, sh, w, code));
}
__device__ __forceinline__ float ll_wait1(Ctx &c, const uint2 *p, uint32_t tag) {
  uint2 v = ll_load1(p);
  Poll w;
  while (v.y != tag) {
    if (poll_expired(c.p, c.sh, w, 400 + (int)(tag & 7)))
      break;
    v = ll_load1(p);
  }
  return __uint_as_float(v.x);
}

// N pairs per lane at once, whole warps: the round trips overlap.  Lanes that want nothing pass any valid pair and !live.
template <int N>
__device__ __forceinline__ void ll_wait(const DecParams &dp, Shared &sh, const uint2 *const (&p)[N], uint32_t tag, float (&out)[N],
                                        bool live = true) {
  Poll w;
  bool ok;
  do {
    uint2 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
      v[i] = ll_load1(p[i]);
    ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      ok = ok && v[i].y == tag;
      out[i] = __uint_as_float(v[i].x);
    }
  } while (!poll_done(dp, sh, w, 400 + (int)(tag & 7), ok || !live));
}

// ---- weight stream ---------------------------------------------------------------------------------------------------
// Ask for the warp's next block (past the end: an empty group, so that the count of groups in flight stays the same).
template <int MODE> __device__ __forceinline__ void request_block(Ctx &c) {
  constexpr bool U4 = MODE == 2;
  if (c.left > 0) {
    const uint32_t dst = c.ring + c.slot * (kDecBlockBytes + (U4 ? kDecScaleBytes : 0)) + c.lane * 16;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst + i * 512), "l"(c.src + i * 512),
                   "l"(c.policy)
                   : "memory");
    if (U4 && c.lane < kDecScaleBytes / 16)
      asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst + kDecBlockBytes),
                   "l"(c.src + kDecBlockBytes), "l"(c.policy)
                   : "memory");
    c.src += kDecBlockBytes + (U4 ? kDecScaleBytes : 0);
    --c.left;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (++c.slot == dec_slots(MODE))
    c.slot = 0;
}
// The oldest block in the ring (slot c.slot): complete for the lane's own pieces, with U4 for the warp.
template <int MODE> __device__ __forceinline__ const uint8_t *wait_block(const Ctx &c) {
  constexpr bool U4 = MODE == 2;
  asm volatile("cp.async.wait_group %0;" ::"n"(dec_slots(MODE) - 1) : "memory");
  if (U4)
    __syncwarp();
  return c.ring_ptr + c.slot * (kDecBlockBytes + (U4 ? kDecScaleBytes : 0));
}

// ---- activations: tagged pairs (or a plain row) -> the operand of the row loops ---------------------------------------
struct XSrc {
  const uint2 *ll;      // tagged source, or null
  const float *plain;   // plain source (the embedding row of layer 0)
  uint32_t tag;
  const float *norm_w;  // RMSNorm weight, or null
};

// A thread takes k = 4i .. 4i+3 for i = tid, tid + 512, ..; kXBatch of them are in flight at a time.  f32 rows: the values
// (times the norm weight) go to shared memory.  int8 and int4: a warp's 32 threads hold 128 k, which get a fixed-point
// scale of their own (one warp reduction, no barrier) and go to planes; `gscale` receives what a group's sums have to be
// multiplied by.  Loops, not straight lines: this code runs 4 L times a token.  Returns the RMSNorm factor.
template <int MODE>
__device__ __forceinline__ float stage_x(Ctx &c, const XSrc &xs, int K, int kind, float *gscale, int *z) {
  const int n4 = K >> 2;
  float ss = 0.f;
#pragma unroll 1
  for (int i0 = c.tid; i0 - c.lane < n4; i0 += kXBatch * kCT) {   // whole warps
    float4 v[kXBatch], nw[kXBatch];
#pragma unroll
    for (int r = 0; r < kXBatch; ++r)
      v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (xs.norm_w != nullptr) {   // depends on nothing: requested before the wait
#pragma unroll
      for (int r = 0; r < kXBatch; ++r)
        if (i0 + r * kCT < n4)
          nw[r] = __ldg(reinterpret_cast<const float4 *>(xs.norm_w) + i0 + r * kCT);
    }
    if (xs.ll == nullptr) {
#pragma unroll
      for (int r = 0; r < kXBatch; ++r)
        if (i0 + r * kCT < n4)
          v[r] = __ldg(reinterpret_cast<const float4 *>(xs.plain) + i0 + r * kCT);
    } else {
      Poll w;
      bool ok;
      do {
        uint4 a[kXBatch], b[kXBatch];
#pragma unroll
        for (int r = 0; r < kXBatch; ++r)
          if (i0 + r * kCT < n4) {
            a[r] = ll_load2(xs.ll + 4 * (i0 + r * kCT));
            b[r] = ll_load2(xs.ll + 4 * (i0 + r * kCT) + 2);
          }
        ok = true;
#pragma unroll
        for (int r = 0; r < kXBatch; ++r)
          if (i0 + r * kCT < n4) {
            ok = ok && a[r].y == xs.tag && a[r].w == xs.tag && b[r].y == xs.tag && b[r].w == xs.tag;
            v[r] = make_float4(__uint_as_float(a[r].x), __uint_as_float(a[r].z), __uint_as_float(b[r].x),
                               __uint_as_float(b[r].z));
          }
      } while (!poll_done(c.p, c.sh, w, 400 + (int)(xs.tag & 7), ok));
    }
#pragma unroll
    for (int r = 0; r < kXBatch; ++r) {
      const int i = i0 + r * kCT;
      if (i - c.lane >= n4)   // warp-uniform
        break;
      if (xs.norm_w != nullptr && i < n4) {
        ss = fmaf(v[r].x, v[r].x, ss);
        ss = fmaf(v[r].y, v[r].y, ss);
        ss = fmaf(v[r].z, v[r].z, ss);
        ss = fmaf(v[r].w, v[r].w, ss);
        v[r] = make_float4(v[r].x * nw[r].x, v[r].y * nw[r].y, v[r].z * nw[r].z, v[r].w * nw[r].w);
      }
      if (MODE >= 1 && kind == B200_W_F32) {
        if (i < n4)
          reinterpret_cast<float4 *>(c.planes)[i] = v[r];
        continue;
      }
      const uint32_t m = 0x7fffffffu;
      const uint32_t mx = __reduce_max_sync(0xffffffffu, max(max(__float_as_uint(v[r].x) & m, __float_as_uint(v[r].y) & m),
                                                             max(__float_as_uint(v[r].z) & m, __float_as_uint(v[r].w) & m)));
      float inv;
      const float scale = fixed_scale(mx, &inv);
      if (c.lane == 0)
        gscale[i >> 5] = inv;
      uint32_t w[4];
      plane_words(fixed_digits(v[r].x, scale), fixed_digits(v[r].y, scale), fixed_digits(v[r].z, scale),
                  fixed_digits(v[r].w, scale), w);
      const int set = i >> 4, e = i & 15;
      // word e of the set's 64 k: int8: k = 16t + 4j; int4: k = 32(j/2) + 8t + 4(j%2)
      const bool i8 = MODE < 2 || kind == B200_W_I8;
      const int t = i8 ? e >> 2 : (e >> 1) & 3, j = i8 ? e & 3 : (e >> 3) * 2 + (e & 1);
      uint8_t *at = c.planes + set * kSet + t * 16 + j * 4;
#pragma unroll
      for (int pl = 0; pl < 4; ++pl)
        *reinterpret_cast<uint32_t *>(at + pl * 64) = w[pl];
      if (!i8) {   // start values of the group's sums
#pragma unroll
        for (int pl = 0; pl < 4; ++pl) {
          const int s = __reduce_add_sync(0xffffffffu, __dp4a((int)w[pl], 0x01010101, 0));
          if (c.lane == pl)
            z[(i >> 5) * 4 + pl] = kFloatBias - 8 * s;
        }
      }
    }
  }
  if (xs.norm_w != nullptr) {
    ss = warp_sum(ss);
    if (c.lane == 0)
      c.sh.redf[c.warp] = ss;
  }
  __syncthreads();
  if (xs.norm_w == nullptr)
    return 1.f;
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < kDecWarps; w += 4) {
    const float4 q = *reinterpret_cast<const float4 *>(&c.sh.redf[w]);
    s += (q.x + q.y) + (q.z + q.w);
  }
  return rsqrtf(s * (1.0f / (float)K) + c.p.eps);
}

// ---- one stream block times the staged activations ---------------------------------------------------------------------
// int8, int4: the planes' sums (f32, each group of 128 k exact); f32: four partial sums.
struct Acc {
  float f[4];
  __device__ __forceinline__ void clear() { f[0] = f[1] = f[2] = f[3] = 0.f; }
};
__device__ __forceinline__ void block_i8(const uint8_t *blk, const uint8_t *planes, float gscale, int lane, Acc &a) {
  const uint8_t *b = planes + lane_at<4>();
  int d[2][4] = {{kFloatBias, kFloatBias, kFloatBias, kFloatBias}, {0, 0, 0, 0}};   // |sums| <= 2^21: see start_u4
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint4 w0 = *reinterpret_cast<const uint4 *>(blk + (s * 64 + lane) * 16);
    const uint4 w8 = *reinterpret_cast<const uint4 *>(blk + (s * 64 + 32 + lane) * 16);
    const uint4 x = *reinterpret_cast<const uint4 *>(b + s * kSet);
    mma_s8(d[s], w0.x, w8.x, w0.y, w8.y, x.x, x.y);
    mma_s8(d[s], w0.z, w8.z, w0.w, w8.w, x.z, x.w);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    a.f[e] = fmaf(__int_as_float(d[0][e] + d[1][e]) - 12582912.0f, gscale, a.f[e]);
}
__device__ __forceinline__ void block_u4(const uint8_t *blk, const uint8_t *planes, const float *gscale, const int *z, int lane,
                                         Acc &a) {
  const uint8_t *b = planes + lane_at<4>();
  const int g = lane >> 2;
  const float2 gs = *reinterpret_cast<const float2 *>(gscale);
  float2 s0 = __half22float2(*reinterpret_cast<const __half2 *>(blk + kDecBlockBytes + g * 4));
  float2 s8 = __half22float2(*reinterpret_cast<const __half2 *>(blk + kDecBlockBytes + (g + 8) * 4));
  s0 = make_float2(s0.x * gs.x, s0.y * gs.y);
  s8 = make_float2(s8.x * gs.x, s8.y * gs.y);
  int d[2][4];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int2 zz = *reinterpret_cast<const int2 *>(z + q * 4 + (lane & 1) * 2);
    d[q][0] = d[q][2] = zz.x;
    d[q][1] = d[q][3] = zz.y;
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {   // two groups of 128 k
    const uint4 w0 = *reinterpret_cast<const uint4 *>(blk + (q * 64 + lane) * 16);
    const uint4 w8 = *reinterpret_cast<const uint4 *>(blk + (q * 64 + 32 + lane) * 16);
    const uint4 x = *reinterpret_cast<const uint4 *>(b + (q * 2) * kSet);
    const uint4 y = *reinterpret_cast<const uint4 *>(b + (q * 2 + 1) * kSet);
    constexpr uint32_t m = 0x0F0F0F0Fu;
    mma_s8(d[q], w0.x & m, w8.x & m, (w0.x >> 4) & m, (w8.x >> 4) & m, x.x, x.y);
    mma_s8(d[q], w0.y & m, w8.y & m, (w0.y >> 4) & m, (w8.y >> 4) & m, x.z, x.w);
    mma_s8(d[q], w0.z & m, w8.z & m, (w0.z >> 4) & m, (w8.z >> 4) & m, y.x, y.y);
    mma_s8(d[q], w0.w & m, w8.w & m, (w0.w >> 4) & m, (w8.w >> 4) & m, y.z, y.w);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      a.f[i] = fmaf(__int_as_float(d[q][i]) - 12582912.0f, i < 2 ? (q ? s0.y : s0.x) : (q ? s8.y : s8.x), a.f[i]);
}
__device__ __forceinline__ void block_f32(const uint8_t *blk, const float *x, int lane, Acc &a) {
  const float *xl = x + (lane >> 4) * 16;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 w = *reinterpret_cast<const float4 *>(blk + (i * 32 + lane) * 16);
    const float4 v = *reinterpret_cast<const float4 *>(xl + 4 * i);
    a.f[i] = fmaf(w.x, v.x, a.f[i]);
    a.f[i] = fmaf(w.y, v.y, a.f[i]);
    a.f[i] = fmaf(w.z, v.z, a.f[i]);
    a.f[i] = fmaf(w.w, v.w, a.f[i]);
  }
}

// ---- one projection ------------------------------------------------------------------------------------------------------
enum { EP_STORE = 0, EP_RESIDUAL = 1, EP_SILU = 2, EP_LOGITS = 3 };
struct Epi {
  int kind;
  uint2 *out;             // tagged output
  uint32_t tag;
  const uint2 *res_ll;    // EP_RESIDUAL: tagged residual vector, or
  const float *res;       // plain
  uint32_t res_tag;
  const float *scale, *bias;   // int8: per row; or null
  const float *next_scale;     // the next layer's
};

// Row data of the epilogue: loaded before the wait for the activations, and in that place (a plain load may be moved).
__device__ __forceinline__ float ld_row(const float *p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// MODE: which weight kinds the model has (0: int8; 1: int8 and f32; 2: all three).
template <int MODE>
__device__ __forceinline__ void gemv_phase(Ctx &c, int ph, const XSrc &xs, const Epi &ep, int layer, float &bestv, int &besti) {
  const DecPhase &q = c.p.phase[ph];
  const int tiles = c.sh.tiles[ph], kind = MODE == 0 ? (int)B200_W_I8 : q.kind;
  if (tiles == 0)
    return;
  // Epilogue: a warp takes tile `warp`, `warp` + 16, ..; two lanes a row (each half of the shares).  What the first tile
  // needs is requested now.
  const int tile0 = c.sh.tile0[ph];
  float e_scale = 1.f, e_bias = 0.f;
  uint2 e_res = make_uint2(0u, 0u);
  auto row_data = [&](int row) {
    if (ep.scale != nullptr)
      e_scale = ld_row(ep.scale + row);
    if (ep.bias != nullptr)
      e_bias = ld_row(ep.bias + row);
    if (ep.res_ll != nullptr)
      e_res = ll_load1(ep.res_ll + row);   // as a rule complete long ago; the tag is checked when it is used
    else if (ep.res != nullptr)
      e_res.x = __float_as_uint(ld_row(ep.res + row));
  };
  if (c.warp < tiles)
    row_data(min((tile0 + c.warp) * kTileRows + (c.lane & 15), q.N - 1));
  if (c.tid == 0 && ep.next_scale != nullptr)   // the next layer's rows: in L2 by then
    prefetch_l2(ep.next_scale + tile0 * kTileRows, 4 * min(tiles * kTileRows, q.N - tile0 * kTileRows));
  float *gscale = reinterpret_cast<float *>(c.planes + (q.K + 127) / 128 * (2 * kSet));
  int *z = reinterpret_cast<int *>(gscale + ((q.K + 255) / 256 * 2 + 3) / 4 * 4);   // int4: start values of the group sums
  const float inv = stage_x<MODE>(c, xs, q.K, kind, gscale, z);
  trace(c, layer, 10 + 4 * ph);
  int b = c.sh.first[ph][c.warp], tile = c.sh.ftile[ph][c.warp], st = b - tile * q.blocks;
  const int b1 = c.sh.first[ph][c.warp + 1];
  Acc a;
  a.clear();
#pragma unroll 1
  for (; b < b1; ++b) {
    const uint8_t *blk = wait_block<MODE>(c);
    if (kind == B200_W_I8)
      block_i8(blk, c.planes + st * (2 * kSet), gscale[st], c.lane, a);
    else if (MODE == 2 && kind == B200_W_U4)
      block_u4(blk, c.planes + st * (4 * kSet), gscale + st * 2, z + st * 8, c.lane, a);
    else if (MODE >= 1)
      block_f32(blk, reinterpret_cast<const float *>(c.planes) + st * 32, c.lane, a);
    if (MODE == 2)
      __syncwarp();   // the scales are read across lanes
    request_block<MODE>(c);
    if (++st == q.blocks || b + 1 == b1) {
      // this warp's share of the tile is complete: rows' sums to shared memory
      float *dst = c.part + (tile + c.warp) * kTileRows;   // (tile, warp) pairs in order: tile + warp is unique
      if (MODE >= 1 && kind == B200_W_F32) {
        float v = (a.f[0] + a.f[1]) + (a.f[2] + a.f[3]);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (c.lane < 16)
          dst[c.lane] = v;
      } else {
        const bool lowp = c.lane & 1;   // odd: planes 2 and 3
        const float f0 = lowp ? 256.f : 16777216.f, f1 = lowp ? 1.f : 65536.f;
        float v0 = fmaf(a.f[0], f0, a.f[1] * f1), v1 = fmaf(a.f[2], f0, a.f[3] * f1);
        v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
        v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
        if ((c.lane & 3) == 0) {
          dst[c.lane >> 2] = v0;
          dst[(c.lane >> 2) + 8] = v1;
        }
      }
      a.clear();
      st = 0;
      ++tile;
    }
  }
  __syncthreads();
  trace(c, layer, 11 + 4 * ph);
  // ---- rows: shares of the warps, epilogue -------------------------------------------------------------------------
#pragma unroll 1
  for (int t = c.warp; t < tiles; t += kDecWarps) {
    const int r = c.lane & 15, row = (tile0 + t) * kTileRows + r;
    const bool in = c.lane < 16 && row < q.N;
    if (t != c.warp)
      row_data(min(row, q.N - 1));
    float v = 0.f;
    const int w1 = c.sh.wlast[ph][t];
#pragma unroll 4
    for (int w = c.sh.wfirst[ph][t] + (c.lane >> 4); w <= w1; w += 2)
      v += c.part[(t + w) * kTileRows + r];
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    v = v * (inv * e_scale) + e_bias;
    if (ep.kind == EP_SILU) {
      const float up = __shfl_down_sync(0xffffffffu, v, 1);   // (gate, up) rows are neighbours
      // (g * sigmoid(g)) * u; e^-g is kept finite (g * 1e-30 is as good a zero as g / inf)
      if (in && (r & 1) == 0)
        ll_store(ep.out + (row >> 1), v * div_normal(1.f, 1.f + fminf(expf(-v), 1e30f)) * up, ep.tag);
    } else if (in) {
      if (ep.kind == EP_LOGITS) {
        c.p.logits[row] = v;
        if (c.p.logits_host != nullptr)
          c.p.logits_host[row] = v;
        if (v > bestv) {   // rows ascend: the first maximum stays
          bestv = v;
          besti = row;
        }
      } else {
        if (ep.res_ll != nullptr && e_res.y != ep.res_tag)
          e_res.x = __float_as_uint(ll_wait1(c, ep.res_ll + row, ep.res_tag));
        ll_store(ep.out + row, __uint_as_float(e_res.x) + v, ep.tag);
      }
    }
  }
  // nobody polls for the next vector before this CTA's own results are out: sixteen warps of polls in the load pipeline
  // stretch the epilogue's loads and shuffles severalfold
  __syncthreads();
  trace(c, layer, 12 + 4 * ph);
}

// ---- attention ---------------------------------------------------------------------------------------------------------
constexpr int kPass = 64;    // keys per pass of a CTA
constexpr int kKRow = D + 4; // a K row in shared memory: 16-byte reads of neighbouring rows hit different banks

template <int G> struct alignas(16) AttnScratch {
  float q[G][D];                    // rotated, scaled by log2(e) / sqrt(D)
  float knew[D], vnew[D];           // this step's K and V rows
  float p[G][kPass];                // probabilities
  float alpha[8], m[8], l[8];       // per head: rescaling of what came before, largest score, sum
  union {
    struct {
      float k[kPass][kKRow];
      float part[8][G][kPass];      // scores over 16 dims each
    };
    float acc[kDecWarps][G][D];
  };
};

// One (kv head, key range) of a layer.  Per pass of 64 keys: a warp loads four K and V rows (16 bytes per lane); scores: a
// lane per key, a warp per (32 keys, 16 dims), so that a K value is read once for all G heads and nothing is reduced across
// lanes; softmax: a warp per head; P*V: a warp its four keys, a lane four dims.  A function of its own: its registers stay
// out of the row loops.
template <int G>
__device__ __noinline__ void attention_range(Shared &sh, const DecLayer *layers, AttnScratch<G> &s, int layer, int pos,
                                             uint32_t layer_tag, long long *tr) {
  const DecParams &p = sh.p;
  const DecLayer &ly = layers[layer];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int par = layer & 1, QD = p.qh * D, KD = p.kvh * D, hk = sh.a_head, sp = sh.a_split, s0 = sh.a_first, s1 = sh.a_end;
  const size_t head = (size_t)hk * p.max_len * D;
  float4 k[4], v[4];
  auto load = [&](float4(&r)[4], const float *cache, int j0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      r[i] = __ldcg(reinterpret_cast<const float4 *>(cache + head + (size_t)min(j0 + i, s1 - 1) * D) + lane);
  };
  load(k, ly.k_cache, s0 + warp * 4);   // the cache does not depend on this layer's q, k, v
  load(v, ly.v_cache, s0 + warp * 4);
  if (layer + 1 < p.L && tid == 0) {   // and the next layer's share of it can come from L2 by then
    const size_t at = head + (size_t)s0 * D;
    prefetch_l2(layers[layer + 1].k_cache + at, (int64_t)(s1 - s0) * D * 4);
    prefetch_l2(layers[layer + 1].v_cache + at, (int64_t)(s1 - s0) * D * 4);
  }
  // ---- q heads (one warp each), then k, then v: (head norm,) rotation ---------------------------------------------
  const uint2 *qkv = p.ll_qkv + (size_t)par * (QD + 2 * KD);
  if (warp < G + 2) {
    const int h = warp;
    const uint2 *src = (h < G ? qkv + (size_t)(hk * G + h) * D : qkv + QD + (h == G ? 0 : KD) + (size_t)hk * D) + lane;
    float in[4];   // dims lane, lane + 32 | lane + 64, lane + 96: rotation pairs (0, 2) and (1, 3)
    ll_wait<4>(p, sh, {src, src + 32, src + 64, src + 96}, layer_tag + T_QKV, in);
    const float *nw = h < G ? ly.q_norm : ly.k_norm;
    if (h <= G && nw != nullptr) {
      const float ss = warp_sum(fmaf(in[0], in[0], in[1] * in[1]) + fmaf(in[2], in[2], in[3] * in[3]));
      const float r = rsqrtf(__fadd_rn(__fmul_rn(ss, 1.0f / (float)D), p.eps));
#pragma unroll
      for (int i = 0; i < 4; ++i)
        in[i] = __fmul_rn(__ldg(nw + lane + 32 * i), __fmul_rn(in[i], r));
    }
    if (h <= G) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float cs = sh.cs[lane + 32 * i], sn = sh.sn[lane + 32 * i], a = in[i], b = in[i + 2];
        in[i] = __fadd_rn(__fmul_rn(a, cs), __fmul_rn(-b, sn));
        in[i + 2] = __fadd_rn(__fmul_rn(b, cs), __fmul_rn(a, sn));
      }
    }
    const float f = h < G ? 0.08838834764831845f * 1.4426950408889634f : 1.f;   // 1/sqrt(128) * log2(e)
    float *dst = (h < G ? s.q[h] : h == G ? s.knew : s.vnew) + lane;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      dst[32 * i] = in[i] * f;
    if (h >= G && s1 == pos + 1) {   // the range that holds the new row writes it
      float *row = (h == G ? ly.k_cache : ly.v_cache) + head + (size_t)pos * D + lane;
      const size_t at = (size_t)(2 * layer + (h == G ? 0 : 1)) * KD + (size_t)hk * D + lane;
      float *stage = p.kv_stage + at;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        row[32 * i] = stage[32 * i] = in[i];
      if (p.rows_host != nullptr)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          p.rows_host[at + 32 * i] = in[i];
    }
  }
  if (tr != nullptr && tid == 0)
    tr[layer * kDecTraceSlots + 1] = clock64();
  float4 acc[G];
#pragma unroll
  for (int g = 0; g < G; ++g)
    acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
  float m = kSeed, l = 0.f;   // of head `warp`
  auto store_k = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4 *>(&s.k[warp * 4 + i][lane * 4]) = k[i];
  };
  // Two barriers per pass: scores of pass i + 1 share a section with P*V of pass i, the K rows of pass i + 1 are stored
  // beside the softmax of pass i.
  store_k();
  if (s0 + kPass < s1)
    load(k, ly.k_cache, s0 + kPass + warp * 4);
  __syncthreads();
#pragma unroll 1
  for (int j0 = s0 - kPass; j0 < s1; j0 += kPass) {
    if (j0 + kPass < s1) {   // scores of the pass at j0 + 64
      const int key = (warp >> 3) * 32 + lane, d0 = (warp & 7) * 16;
      const float *kr = (j0 + kPass + key == pos ? s.knew : s.k[key]) + d0;
      float sc[G];
#pragma unroll
      for (int g = 0; g < G; ++g)
        sc[g] = 0.f;
#pragma unroll 2
      for (int i = 0; i < 16; i += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(kr + i);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float4 y = *reinterpret_cast<const float4 *>(&s.q[g][d0 + i]);
          sc[g] = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, sc[g]))));
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g)
        s.part[warp & 7][g][key] = sc[g];
    }
    if (j0 >= s0) {   // P*V of the pass at j0
      if (pos >= j0 + warp * 4 && pos < j0 + warp * 4 + 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (j0 + warp * 4 + i == pos)
            v[i] = *reinterpret_cast<const float4 *>(&s.vnew[lane * 4]);
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 pg = *reinterpret_cast<const float4 *>(&s.p[g][warp * 4]);
        const float ag = s.alpha[g];
        acc[g].x = fmaf(pg.x, v[0].x, fmaf(pg.y, v[1].x, fmaf(pg.z, v[2].x, fmaf(pg.w, v[3].x, acc[g].x * ag))));
        acc[g].y = fmaf(pg.x, v[0].y, fmaf(pg.y, v[1].y, fmaf(pg.z, v[2].y, fmaf(pg.w, v[3].y, acc[g].y * ag))));
        acc[g].z = fmaf(pg.x, v[0].z, fmaf(pg.y, v[1].z, fmaf(pg.z, v[2].z, fmaf(pg.w, v[3].z, acc[g].z * ag))));
        acc[g].w = fmaf(pg.x, v[0].w, fmaf(pg.y, v[1].w, fmaf(pg.z, v[2].w, fmaf(pg.w, v[3].w, acc[g].w * ag))));
      }
      if (j0 + kPass >= s1)
        break;
      load(v, ly.v_cache, j0 + kPass + warp * 4);
    }
    __syncthreads();
    if (j0 + 2 * kPass < s1) {
      store_k();
      if (j0 + 3 * kPass < s1)
        load(k, ly.k_cache, j0 + 3 * kPass + warp * 4);
    }
    if (warp < G) {   // softmax of the pass at j0 + 64
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        a += s.part[i][warp][lane];
        b += s.part[i][warp][lane + 32];
      }
      a = j0 + kPass + lane < s1 ? a : -INFINITY;
      b = j0 + kPass + lane + 32 < s1 ? b : -INFINITY;
      const float nm = fmaxf(m, warp_max(fmaxf(a, b)));
      const float al = ex2(m - nm);
      a = ex2(a - nm);
      b = ex2(b - nm);
      m = nm;
      l = fmaf(l, al, warp_sum(a + b));
      s.p[warp][lane] = a;
      s.p[warp][lane + 32] = b;
      if (lane == 0) {
        s.alpha[warp] = al;
        s.m[warp] = m;
        s.l[warp] = l;
      }
    }
    __syncthreads();
  }
  if (tr != nullptr && tid == 0)
    tr[layer * kDecTraceSlots + 2] = clock64();
  // ---- the warps' sums (acc takes the place of k and part: everybody is past them) -----------------------------------
#pragma unroll
  for (int g = 0; g < G; ++g)
    *reinterpret_cast<float4 *>(&s.acc[warp][g][lane * 4]) = acc[g];
  __syncthreads();
#pragma unroll 1
  for (int o = tid; o < G * D; o += kCT) {
    const int g = o >> 7, d = o & (D - 1), h = hk * G + g;
    float a = 0.f;
#pragma unroll 8
    for (int w = 0; w < kDecWarps; ++w)
      a += s.acc[w][g][d];
    if (sh.splits == 1) {
      ll_store(p.ll_attn + (size_t)par * QD + h * D + d, div_normal(a, s.l[g]), layer_tag + T_ATTN);
    } else {
      uint2 *part = p.ll_part + (((size_t)par * p.qh + h) * kDecMaxSplits + sp) * (D + 2);
      ll_store(part + d, a, layer_tag + T_PART);
      if (d < 2)
        ll_store(part + D + d, d == 0 ? s.m[g] : s.l[g], layer_tag + T_PART);
    }
  }
  if (tr != nullptr && tid == 0)
    tr[layer * kDecTraceSlots + 3] = clock64();
}

template <int G> __device__ __forceinline__ void attention_phase(Ctx &c, int layer, int pos) {
  const DecParams &p = c.p;
  if (c.sh.a_head >= 0)
    attention_range<G>(c.sh, c.layers, *reinterpret_cast<AttnScratch<G> *>(c.planes), layer, pos, tag_of(c, layer, 0), c.tr);
  // ---- fold the ranges: one warp per four outputs, one lane per range ---------------------------------------------------
  if (c.sh.splits > 1) {
    const int par = layer & 1, o1 = c.sh.out1;
#pragma unroll 1
    for (int o = (c.sh.out0 + c.warp) * 4; o < o1 * 4; o += kDecWarps * 4) {
      const bool live = c.lane < c.sh.splits;
      const uint2 *part = p.ll_part + (((size_t)par * p.qh + (o >> 7)) * kDecMaxSplits + (live ? c.lane : 0)) * (D + 2);
      float in[6];
      Poll w;
      const uint32_t tag = tag_of(c, layer, T_PART);
      bool ok;
      do {
        const uint4 v[3] = {ll_load2(part + (o & (D - 1))), ll_load2(part + (o & (D - 1)) + 2), ll_load2(part + D)};
        ok = true;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          ok = ok && v[i].y == tag && v[i].w == tag;
          in[2 * i] = __uint_as_float(v[i].x);
          in[2 * i + 1] = __uint_as_float(v[i].z);
        }
      } while (!poll_done(p, c.sh, w, 400 + (int)(tag & 7), ok));
      if (!live)
        in[4] = kSeed;
      const float b = ex2(in[4] - warp_max(in[4]));
      const float L = warp_sum(in[5] * b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float A = warp_sum(in[i] * b);
        if (c.lane == i)
          ll_store(p.ll_attn + (size_t)par * p.qh * D + o + i, div_normal(A, L), tag_of(c, layer, T_ATTN));
      }
    }
    __syncthreads();   // as at the end of a projection
  }
  trace(c, layer, 4);
}

} // namespace

template <int G, int MODE>
__global__ void __launch_bounds__(kDecThreads, 1) decode_step_kernel(const __grid_constant__ DecParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  // layout: Shared | layer table | planes, f32 vector / attention scratch | partial sums | rings
  Shared &sh = *reinterpret_cast<Shared *>(smem);
  uint8_t *at = smem + (sizeof(Shared) + 127) / 128 * 128;
  DecLayer *layers = reinterpret_cast<DecLayer *>(at);
  at += ((size_t)p.L * sizeof(DecLayer) + 127) / 128 * 128;
  uint8_t *planes = at;
  at += p.union_bytes;
  float *part = reinterpret_cast<float *>(at);
  at += p.part_rows * kTileRows * 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kBlock = kDecBlockBytes + (MODE == 2 ? kDecScaleBytes : 0);
  uint8_t *ring = at + (size_t)warp * dec_slots(MODE) * kBlock;

  Ctx c{p, sh, layers, planes, part, smem_u32(ring), ring,
        p.stream + p.warp_off[blockIdx.x * kDecWarps + warp] + lane * 16, 0, 0, 0ull, (int)threadIdx.x, lane, warp,
        ((uint32_t)p.state[4] + 1u) * (8u * (uint32_t)(p.L + 3)),
        (p.trace != nullptr && blockIdx.x % p.trace_stride == 0)
            ? p.trace + (size_t)(blockIdx.x / p.trace_stride) * (p.L + 1) * kDecTraceSlots
            : nullptr};
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(c.policy));
  const int token = p.state[0], pos = p.state[1];
  // blocks of this warp over the whole token
#pragma unroll 1
  for (int i = 0; i < 5; ++i) {
    const int t0 = share_begin(p.phase[i].tiles, blockIdx.x, gridDim.x);
    const int n = share_begin(p.phase[i].tiles, blockIdx.x + 1, gridDim.x) - t0, nb = n * p.phase[i].blocks;
    if (threadIdx.x == 0) {
      sh.tile0[i] = t0;
      sh.tiles[i] = n;
    }
    const int b0 = warp_begin(nb, warp), b1 = warp_begin(nb, warp + 1);
    c.left += (b1 - b0) * (i < 4 ? p.L : 1);
    if (lane == 0) {
      sh.first[i][warp] = b0;
      sh.ftile[i][warp] = b0 / p.phase[i].blocks;
      if (warp == kDecWarps - 1)
        sh.first[i][kDecWarps] = nb;
    }
    if ((int)threadIdx.x < n) {
      const int b = threadIdx.x * p.phase[i].blocks, e = b + p.phase[i].blocks - 1;
      sh.wfirst[i][threadIdx.x] = (uint8_t)warp_of(nb, b);
      sh.wlast[i][threadIdx.x] = (uint8_t)warp_of(nb, e);
    }
  }
#pragma unroll 1
  for (int s = 0; s < dec_slots(MODE); ++s)   // fill the ring
    request_block<MODE>(c);
  for (int i = threadIdx.x; i < (int)(sizeof(DecParams) / 4); i += kCT)
    reinterpret_cast<uint32_t *>(&sh.p)[i] = reinterpret_cast<const uint32_t *>(&p)[i];
  if (threadIdx.x == 0) {
    sh.abort_flag = 0;
    // key ranges per kv head: one pass of the sixteen warps (64 keys) each, as long as they fit the CTAs and the lanes
    // that fold them; the (head, range) items are spread over the CTAs
    const int len = pos + 1, S = min(min(kDecMaxSplits, (int)gridDim.x / p.kvh), (len + 63) / 64), items = p.kvh * S;
    const int item = (int)((blockIdx.x * items + gridDim.x - 1) / gridDim.x);
    const bool has = item < items && item * gridDim.x / items == blockIdx.x;
    const int hk = item / S, sp = item - hk * S, chunk = (len + S - 1) / S;
    sh.splits = S;
    sh.a_head = has ? hk : -1;
    sh.a_split = sp;
    sh.a_first = sp * chunk;
    sh.a_end = min(len, (sp + 1) * chunk);
    sh.out0 = share_begin(p.qh * D / 4, blockIdx.x, gridDim.x);
    sh.out1 = share_begin(p.qh * D / 4, blockIdx.x + 1, gridDim.x);
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < p.L * (int)(sizeof(DecLayer) / 8); i += kCT)
    reinterpret_cast<uint64_t *>(layers)[i] = __ldg(reinterpret_cast<const unsigned long long *>(p.layers) + i);
  if (threadIdx.x < D / 2) {
    // subgraph0_decode_simplify.mlir:52-59
    const float th = __fmul_rn(__ldg(p.inv_freq + threadIdx.x), (float)pos);
    sh.cs[threadIdx.x] = cosf(th);
    sh.sn[threadIdx.x] = sinf(th);
  }
  __syncthreads();

  const int H = p.H, QD = p.qh * D, KD = p.kvh * D;
  const float *embed_row = p.embed + (size_t)token * H;
  float bestv = -INFINITY;
  int besti = 0x7fffffff;
  // step 0..3 of layer l = q|k|v (and attention), o, gate|up, down; layer L has the lm_head only
#pragma unroll 1
  for (int n = 0; n <= 4 * p.L; ++n) {
    const int l = n >> 2, step = l == p.L ? 4 : n & 3, par = l & 1;
    const DecLayer *ly = layers + (l < p.L ? l : 0), *nx = layers + (l + 1 < p.L ? l + 1 : 0);
    // residual stream entering the layer: the embedding row, or layer l-1's output
    const uint2 *xin = l == 0 ? nullptr : p.ll_xa + (size_t)(par ^ 1) * H;
    const uint32_t xin_tag = tag_of(c, l - 1, T_XA);
    uint2 *xb = p.ll_xb + (size_t)par * H, *mid = p.ll_mid + (size_t)par * p.F;
    XSrc xs;
    Epi ep;
    switch (step) {
    case 0:   // q | k | v (+ bias) <- RMSNorm(x)
      xs = XSrc{xin, embed_row, xin_tag, ly->in_norm};
      ep = Epi{EP_STORE, p.ll_qkv + (size_t)par * (QD + 2 * KD), tag_of(c, l, T_QKV), nullptr, nullptr, 0u, ly->scale[0],
               ly->qkv_bias, nx->scale[0]};
      break;
    case 1:   // x1 = x + attn @ Wo
      xs = XSrc{p.ll_attn + (size_t)par * QD, nullptr, tag_of(c, l, T_ATTN), nullptr};
      ep = Epi{EP_RESIDUAL, xb, tag_of(c, l, T_XB), xin, l == 0 ? embed_row : nullptr, xin_tag, ly->scale[1], nullptr,
               nx->scale[1]};
      break;
    case 2:   // silu(gate) * up <- RMSNorm(x1)
      xs = XSrc{xb, nullptr, tag_of(c, l, T_XB), ly->post_norm};
      ep = Epi{EP_SILU, mid, tag_of(c, l, T_MID), nullptr, nullptr, 0u, ly->scale[2], nullptr, nx->scale[2]};
      break;
    case 3:   // x2 = x1 + mid @ Wdown
      xs = XSrc{mid, nullptr, tag_of(c, l, T_MID), nullptr};
      ep = Epi{EP_RESIDUAL, p.ll_xa + (size_t)par * H, tag_of(c, l, T_XA), xb, nullptr, tag_of(c, l, T_XB), ly->scale[3],
               nullptr, nx->scale[3]};
      break;
    default:  // logits <- RMSNorm(x) @ lm_head
      xs = XSrc{xin, embed_row, xin_tag, p.final_norm};
      ep = Epi{EP_LOGITS, nullptr, 0u, nullptr, nullptr, 0u, p.lm_scale, nullptr, nullptr};
      break;
    }
    trace(c, l, 5 + step);
    gemv_phase<MODE>(c, step, xs, ep, l, bestv, besti);
    if (step == 0) {
      trace(c, l, 0);
      if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {   // the next layer's norm weights and bias: in L2 by then
        prefetch_l2(nx->in_norm, 4 * H);
        prefetch_l2(nx->post_norm, 4 * H);
        if (nx->qkv_bias != nullptr)
          prefetch_l2(nx->qkv_bias, 4 * (QD + 2 * KD));
      }
      attention_phase<G>(c, l, pos);
    }
  }

  // ---- greedy token (Sampler.h:101-104: first maximum) -------------------------------------------------------------
  auto better = [&](float v, int i) {
    if (v > bestv || (v == bestv && i < besti)) {
      bestv = v;
      besti = i;
    }
  };
  auto warp_best = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      better(__shfl_xor_sync(0xffffffffu, bestv, o), __shfl_xor_sync(0xffffffffu, besti, o));
  };
  warp_best();
  if (lane == 0) {
    sh.bestv[warp] = bestv;
    sh.besti[warp] = besti;
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t ctag = tag_of(c, p.L, T_CAND);
    bestv = sh.bestv[lane & (kDecWarps - 1)];
    besti = sh.besti[lane & (kDecWarps - 1)];
    warp_best();
    if (lane == 0) {
      ll_store(p.ll_cand + 2 * blockIdx.x, bestv, ctag);
      ll_store(p.ll_cand + 2 * blockIdx.x + 1, __int_as_float(besti), ctag);
    }
    if (blockIdx.x == 0) {
      bestv = -INFINITY;
      besti = 0x7fffffff;
      for (int i = 0; i < (int)gridDim.x; i += 32) {
        const bool live = i + lane < (int)gridDim.x;
        const uint2 *cand = p.ll_cand + 2 * (live ? i + lane : 0);
        float in[2];
        ll_wait<2>(p, sh, {cand, cand + 1}, ctag, in, live);
        if (live)
          better(in[0], __float_as_int(in[1]));
      }
      __syncwarp();
      warp_best();
      if (lane == 0 && sh.abort_flag == 0) {
        const int next = besti == 0x7fffffff ? 0 : besti;
        const int cnt = p.state[3];
        if (cnt < p.history_cap)
          p.history[cnt] = next;
        p.state[3] = cnt + 1;
        p.state[2] = next;
        p.state[0] = next;
        p.state[1] = pos + 1;
        p.state[4] = p.state[4] + 1;   // launches completed (base of the tags)
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");   // (an abandoned step may still have copies in flight)
}

// ---- stream builder: packed rows of one projection -> the warps' blocks ---------------------------------------------
// One CTA per block: 16 rows of a tile, one step of k, in the order the lanes read them.  chunk (16 bytes) c of a block:
//   int8: set s = c/64 (64 k), row (c%64)/32*8 + lane/4, k = 64 s + 16 (lane%4) ..+15
//   int4: group q = c/64 (128 k), row as above; word i, byte e: low nibble k = 128 q + 32 i + 8 (lane%4) + e, high + 4
//   f32:  row lane%16, k = 16 (lane/16) + 4 (c/32) ..+3
__global__ void dec_build_kernel(const uint8_t *rows, const void *scale, int scale_dtype, int group, int64_t row_bytes,
                                 DecPhase ph, int grid_ctas, int block_bytes, const int64_t *warp_off, const int64_t *skip,
                                 uint8_t *stream) {
  const int tile = blockIdx.x / ph.blocks, st = blockIdx.x - tile * ph.blocks;
  // owner: the CTA whose contiguous share of the tiles holds this one, the warp whose share of its blocks does
  int cta = (int)(((int64_t)tile * grid_ctas) / ph.tiles);
  while (share_begin(ph.tiles, cta + 1, grid_ctas) <= tile)
    ++cta;
  while (share_begin(ph.tiles, cta, grid_ctas) > tile)
    --cta;
  const int t0 = share_begin(ph.tiles, cta, grid_ctas), nb = (share_begin(ph.tiles, cta + 1, grid_ctas) - t0) * ph.blocks;
  const int b = (tile - t0) * ph.blocks + st, w = warp_of(nb, b);
  const int at = cta * kDecWarps + w;
  uint8_t *dst = stream + warp_off[at] + skip[at] + (int64_t)(b - warp_begin(nb, w)) * block_bytes;
  const int ck = threadIdx.x, lane = ck & 31;   // 128 threads = 128 chunks
  const int r16 = ph.kind == B200_W_F32 ? lane & 15 : ((ck >> 5) & 1) * 8 + (lane >> 2);
  const int64_t row = (int64_t)tile * kTileRows + r16;
  uint32_t out[4] = {0u, 0u, 0u, 0u};
  if (row < ph.N) {
    const uint8_t *src = rows + row * row_bytes;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // four consecutive k are neighbours in a packed row
      if (ph.kind == B200_W_I8) {
        const int k = st * 128 + (ck >> 6) * 64 + (lane & 3) * 16 + 4 * i;
        if (k < ph.K)
          out[i] = *reinterpret_cast<const uint32_t *>(src + packed_offset(B200_W_I8, ph.K, k, nullptr));
      } else if (ph.kind == B200_W_U4) {
        const int k = st * 256 + (ck >> 6) * 128 + 32 * i + (lane & 3) * 8;   // K is a multiple of 256
        for (int h = 0; h < 2; ++h) {
          const uint32_t v = *reinterpret_cast<const uint16_t *>(src + packed_offset(B200_W_U4, ph.K, k + 4 * h, nullptr));
          out[i] |= ((v & 0xFu) | (v & 0xF0u) << 4 | (v & 0xF00u) << 8 | (v & 0xF000u) << 12) << (4 * h);
        }
      } else {
        const int k = st * 32 + (lane >> 4) * 16 + 4 * (ck >> 5) + i;
        out[i] = *reinterpret_cast<const uint32_t *>(src + packed_offset(B200_W_F32, ph.K, k, nullptr));
      }
    }
  }
  *reinterpret_cast<uint4 *>(dst + ck * 16) = make_uint4(out[0], out[1], out[2], out[3]);
  if (ph.kind == B200_W_U4 && ck < 32) {   // scales [row][group] behind the weights
    const int64_t r = (int64_t)tile * kTileRows + (ck >> 1);
    __half h = __float2half_rn(0.f);
    if (r < ph.N)
      h = __float2half_rn(load_as_float(scale, scale_dtype,
                                        group ? r * (ph.K / 128) + st * 2 + (ck & 1) : r));
    *reinterpret_cast<__half *>(dst + kDecBlockBytes + ck * 2) = h;
  }
}

int dec_block_k(int kind) { return kind == B200_W_I8 ? 128 : kind == B200_W_U4 ? 256 : 32; }

int dec_build_phase(const b200_weight *w, const DecPhase &ph, int grid, int block_bytes, const int64_t *warp_off,
                    const int64_t *skip, uint8_t *stream, cudaStream_t st) {
  const bool grouped = w->kind == B200_W_U4 && w->group > 0 && w->group < w->K;
  dec_build_kernel<<<ph.tiles * ph.blocks, 128, 0, st>>>((const uint8_t *)w->w, w->scale, w->scale_dtype, grouped ? 1 : 0,
                                                         packed_row_bytes(w->kind, w->K), ph, grid, block_bytes, warp_off,
                                                         skip, stream);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

size_t dec_union_bytes(const DecPhase *ph, int G) {
  size_t n = 0;
  switch (G) {
#define B200_G(G_) case G_: n = sizeof(AttnScratch<G_>); break;
    B200_G(1) B200_G(2) B200_G(3) B200_G(4) B200_G(6) B200_G(8)
#undef B200_G
  default: break;
  }
  for (int i = 0; i < 5; ++i) {
    const size_t groups = (size_t)(ph[i].K + 255) / 256 * 2;   // planes, scale and start values of 128 k
    n = std::max(n, ph[i].kind == B200_W_F32 ? (size_t)ph[i].K * 4 : groups * (2 * kSet + 4 + 16) + 16);
  }
  return (n + 127) / 128 * 128;
}
// Which weight kinds the kernel has to be compiled for: 0: int8; 1: int8 and f32; 2: all three.
static int dec_mode(const DecPhase *ph) {
  int mode = 0;
  for (int i = 0; i < 5; ++i)
    mode = std::max(mode, ph[i].kind == B200_W_U4 ? 2 : ph[i].kind == B200_W_F32 ? 1 : 0);
  return mode;
}
size_t dec_shared_bytes(const DecParams &p) {
  return (sizeof(Shared) + 127) / 128 * 128 + ((size_t)p.L * sizeof(DecLayer) + 127) / 128 * 128 +
         p.union_bytes + (size_t)p.part_rows * kTileRows * 4 +
         (size_t)kDecWarps * dec_slots(dec_mode(p.phase)) * p.block_bytes;
}
bool dec_group_built(int G) { return G == 1 || G == 2 || G == 3 || G == 4 || G == 6 || G == 8; }

int dec_launch(const DecParams &p, int grid, size_t smem, cudaStream_t st) {
  const void *kern = nullptr;
  const int mode = dec_mode(p.phase);
  const int G = p.qh / p.kvh;
  switch (G) {
#define B200_G(G_)                                                                                                     \
  case G_:                                                                                                             \
    kern = mode == 0 ? (const void *)decode_step_kernel<G_, 0>                                                         \
         : mode == 1 ? (const void *)decode_step_kernel<G_, 1> : (const void *)decode_step_kernel<G_, 2>;              \
    break;
    B200_G(1) B200_G(2) B200_G(3) B200_G(4) B200_G(6) B200_G(8)
#undef B200_G
  default: return fail(B200_EINVAL, "decode kernel: group size %d not built", G);
  }
  static RaisedOn raised[9][3];
  if (int rc = raise_shared_limit(raised[G][mode], kern, 227 * 1024))
    return rc;
  void *args[] = {(void *)&p};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs co-resident, or the launch fails
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  B200_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
  count_launch();
  return B200_OK;
}

} // namespace b200
