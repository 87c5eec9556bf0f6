// b200_gemv for int8 and int4 weights, M = 1..16 activation rows: see gemv_mma.cuh for the arithmetic.
//
// A warp takes a tile of 16 output rows (or, for narrow projections, a share of the tile's k: `ks` warps of the CTA meet
// in shared memory); one CTA per SM stages the planes of all activation rows once and walks over its tiles.  The weights
// of the next step (eight 16-byte loads per lane, 64 KB per SM) are in flight while a step is multiplied, the first
// step's already while the activations are staged.
//
// Bound: HBM for one row (int8 lm_head 151936 x 1536: 42 us, 5.6 TB/s; int4 152000 x 4096: 70 us; the FFMA kernel: 50 and
// 111 us), the shared-memory reads and MMAs of four columns per activation row for many (int4 14336 x 4096, 5 rows: 130 ->
// 27 us; 16 rows: 363 -> 61 us), and for short calls the chain launch - first load - quantise - first step - sum.
#include "gemv_mma.cuh"

#include <mutex>

namespace b200 {

struct MmaP {
  const void *x;
  const uint8_t *w;
  const void *scale;
  const float *bias, *residual, *norm_w;
  void *y;
  int64_t x_ld, y_ld, row_bytes;
  int K, Kp, N, M;
  int units;          // 16-byte units per row the MMA steps cover (int4: whole 1024-element blocks)
  int tail_k0, tunits; // int4: first k of the short last block, and its units (0: none)
  int steps, slab_steps, slab_k;
  int x_dtype, y_dtype, scale_dtype, x_vec;
  int ngroups, scale_vec;
  int accumulate, silu_pairs;
  int reg_x;          // one activation row that fits the threads' registers
  int ks, slots, tiles, rounds;
  int start_off, tail_off, tstart_off, part_off, red_off;   // shared-memory layout (bytes)
  float eps;
};

template <bool XF> __device__ __forceinline__ float4 act4(const MmaP &p, int m, int k) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  const int64_t at = (int64_t)m * p.x_ld + k;
  if (XF) {
    if (k < p.K)
      v = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p.x) + at));
  } else if (p.x_vec && k + 4 <= p.K) {
    const uint2 h = __ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(p.x) + at));
    float2 a, b;
    if (p.x_dtype == B200_F16) {
      a = __half22float2(*reinterpret_cast<const __half2 *>(&h.x));
      b = __half22float2(*reinterpret_cast<const __half2 *>(&h.y));
    } else {
      a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&h.x));
      b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&h.y));
    }
    v = make_float4(a.x, a.y, b.x, b.y);
  } else {
    if (k < p.K) v.x = load_as_float(p.x, p.x_dtype, at);
    if (k + 1 < p.K) v.y = load_as_float(p.x, p.x_dtype, at + 1);
    if (k + 2 < p.K) v.z = load_as_float(p.x, p.x_dtype, at + 2);
    if (k + 3 < p.K) v.w = load_as_float(p.x, p.x_dtype, at + 3);
  }
  return v;
}
template <bool XF> __device__ __forceinline__ float4 normed(const MmaP &p, int k, float4 v) {
  if (p.norm_w != nullptr) {
    if (XF) {
      if (k < p.K) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(p.norm_w + k));
        v = make_float4(v.x * w.x, v.y * w.y, v.z * w.z, v.w * w.w);
      }
    } else {
      if (k < p.K) v.x *= __ldg(p.norm_w + k);
      if (k + 1 < p.K) v.y *= __ldg(p.norm_w + k + 1);
      if (k + 2 < p.K) v.z *= __ldg(p.norm_w + k + 2);
      if (k + 3 < p.K) v.w *= __ldg(p.norm_w + k + 3);
    }
  }
  return v;
}
__device__ __forceinline__ uint32_t absbits4(float4 v) {
  const uint32_t m = 0x7fffffffu;
  return max(max(__float_as_uint(v.x) & m, __float_as_uint(v.y) & m),
             max(__float_as_uint(v.z) & m, __float_as_uint(v.w) & m));
}

// The eight f16 group scales of a block, for the rows of a tile.
struct Scales {
  uint4 s0, s8;
};
__device__ __forceinline__ uint4 block_scales(const MmaP &p, int64_t row, int b) {
  const __half *s = reinterpret_cast<const __half *>(p.scale) + row * p.ngroups + b * 8;
  if (p.scale_vec)
    return __ldg(reinterpret_cast<const uint4 *>(s));
  const uint16_t *h = reinterpret_cast<const uint16_t *>(s);
  uint4 v;
  v.x = __ldg(h) | (uint32_t)__ldg(h + 1) << 16;
  v.y = __ldg(h + 2) | (uint32_t)__ldg(h + 3) << 16;
  v.z = __ldg(h + 4) | (uint32_t)__ldg(h + 5) << 16;
  v.w = __ldg(h + 6) | (uint32_t)__ldg(h + 7) << 16;
  return v;
}

// The whole product in f32, for calls with a row whose bulk lies too far below its largest elements for four digits (a channel
// some thousand times the rest): the output columns that do not use those channels would lose (10000 times: 4.8e-6 of their
// size, here 1.4e-7).  A warp takes a pair of output rows and four activation rows at a time, lanes the units.  Small and out
// of line: the code of the products above must stay short.
template <int KIND, bool GROUPED, bool XF>
__device__ __noinline__ void float_rows(const MmaP &p, const float *s_scale, const float *s_inv) {
  constexpr bool U4 = KIND == B200_W_U4;
  const int lane = threadIdx.x & 31, W = blockDim.x >> 5, E = U4 ? 32 : 16, units = p.Kp / E;
#pragma unroll 1
  for (int64_t n0 = 2 * ((int64_t)blockIdx.x * W + (threadIdx.x >> 5)); n0 < p.N; n0 += 2 * (int64_t)gridDim.x * W)
#pragma unroll 1
    for (int m0 = 0; m0 < p.M; m0 += 4) {
      float acc[2][4] = {};
#pragma unroll 1
      for (int u = lane; u < units; u += 32) {
        const int b = u >> 5, nu = min(32, units - 32 * b);   // packed rows: blocks of 32 units, see packed_offset
        uint4 w[2];
#pragma unroll
        for (int r = 0; r < 2; ++r)
          w[r] = ld_weights(p.w + min(n0 + r, (int64_t)p.N - 1) * p.row_bytes + (int64_t)u * 16);
#pragma unroll 1
        for (int j = 0; j < (U4 ? 8 : 4); ++j) {
          const int k = b * 32 * E + j * (nu * 4) + 4 * (u & 31);
          float q[2][4];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint32_t a = U4 ? w[r].x & 0xFFFFu : w[r].x;   // this group's four weights
            float g = 1.f;
            if (GROUPED && k < p.K)
              g = __half2float(__ldg(reinterpret_cast<const __half *>(p.scale) + min(n0 + r, (int64_t)p.N - 1) * p.ngroups + (k >> 7)));
#pragma unroll
            for (int e = 0; e < 4; ++e)
              q[r][e] = g * (float)(U4 ? (int)(a >> (4 * e) & 15u) - 8 : (int)(int8_t)(a >> (8 * e)));
            if (U4 && !(j & 1)) {   // the next group: the upper half of the word, or the next word
              w[r].x >>= 16;
            } else {
              w[r] = make_uint4(w[r].y, w[r].z, w[r].w, 0u);
            }
          }
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const float4 x = normed<XF>(p, k, act4<XF>(p, min(m0 + m, p.M - 1), k));
#pragma unroll
            for (int r = 0; r < 2; ++r)
              acc[r][m] += fmaf(x.x, q[r][0], fmaf(x.y, q[r][1], fmaf(x.z, q[r][2], x.w * q[r][3])));
          }
        }
      }
      float mine = 0.f;   // lane 2m + r: row n0 + r, activation row m0 + m
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float v = warp_sum(acc[r][m]);
          if (lane == 2 * m + r)
            mine = v;
        }
      const int m = m0 + (lane >> 1);
      const int64_t row = n0 + (lane & 1);
      const bool in = lane < 8 && m < p.M && row < p.N;
      float v = mine;
      if (in) {
        v *= s_inv[m] * s_scale[m];   // 1, the RMSNorm's factor, or NaN
        if (!GROUPED)
          v *= load_as_float(p.scale, p.scale_dtype, row);
        if (p.bias != nullptr)
          v = __ldg(p.bias + row) + v;
      }
      const float up = __shfl_down_sync(0xffffffffu, v, 1);
      int64_t o = (int64_t)m * p.y_ld + row;
      if (!in || (p.silu_pairs && (lane & 1)))
        continue;
      if (p.silu_pairs) {
        v = silu_gate(v, up);
        o = (int64_t)m * p.y_ld + (row >> 1);
      } else if (p.residual != nullptr) {
        v = p.residual[o] + v;
      }
      if (p.y_dtype == B200_F32)
        ((float *)p.y)[o] = p.accumulate ? ((float *)p.y)[o] + v : v;
      else
        ((__half *)p.y)[o] = __float2half_rn(p.accumulate ? __half2float(((__half *)p.y)[o]) + v : v);
    }
}

template <int COLS> constexpr int kMaxWarps = COLS <= 16 ? 16 : COLS <= 32 ? 12 : 8;   // what the accumulators leave registers for

// XF: f32 activations in whole 16-byte groups.  Compiled for the two common cases so that the code a short call has to
// fetch stays small: a GEMV of a few microseconds is bound by its chain of latencies (instruction fetch among them).
template <int KIND, int COLS, bool GROUPED, bool XF>
__global__ void __launch_bounds__(kMaxWarps<COLS> * 32, 1) gemv_mma_kernel(const __grid_constant__ MmaP p) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x, W = nthr >> 5;
  uint8_t *planes = sm;
  int *start = reinterpret_cast<int *>(sm + p.start_off);
  uint8_t *tplanes = sm + p.tail_off;
  int *tstart = reinterpret_cast<int *>(sm + p.tstart_off);
  float *part = reinterpret_cast<float *>(sm + p.part_off);      // [2][slots][ks][M][16]
  uint32_t *red = reinterpret_cast<uint32_t *>(sm + p.red_off);  // [M][W]
  float *redf = reinterpret_cast<float *>(red + p.M * W);        // [M][W]
  uint32_t *redb = reinterpret_cast<uint32_t *>(redf + p.M * W); // [M][W]
  float *s_scale = reinterpret_cast<float *>(redb + p.M * W), *s_inv = s_scale + p.M;   // [M] each
  __shared__ int s_wide;                                         // some row has too little of itself in four digits
  const int slot = warp / p.ks, kp = warp - slot * p.ks;
  const int steps = p.steps;
  constexpr bool U4 = KIND == B200_W_U4;
  const int nu = p.tunits;   // int4: units of the short last block
  const bool one_slab = p.slab_steps >= p.steps;

  // (warps beyond the slots only help with the staging)
  auto tile_of = [&](int r) { return slot < p.slots ? ((int64_t)r * gridDim.x + blockIdx.x) * p.slots + slot : (int64_t)p.tiles; };
  TileRows rows{};
  uint4 w[8];
  Scales sc{};
  auto fetch = [&](int64_t tile, const TileRows &tr, int s, uint4(&dst)[8], Scales &ds) {
    load_step(tr, s, p.units, dst);
    if constexpr (U4 && GROUPED) {
      const int64_t ra = min(tile * kTileRows + (lane >> 2), (int64_t)p.N - 1);
      const int64_t rb = min(tile * kTileRows + (lane >> 2) + 8, (int64_t)p.N - 1);
      ds.s0 = block_scales(p, ra, s >> 1);
      ds.s8 = block_scales(p, rb, s >> 1);
    }
  };
  if (tile_of(0) < p.tiles && kp < steps) {
    rows = tile_rows(p.w, p.row_bytes, tile_of(0) * kTileRows, p.N);
    fetch(tile_of(0), rows, kp, w, sc);
  }

  // ---- activations: largest magnitude (and mean square, for the RMSNorm) of every row, then the planes ------------
  // Group i of a row (4 consecutive k; int4: two such 16 apart) -> its first k.
  auto k_of = [&](int i, int units) { return U4 ? group_u4(i).k : group_i8(i, units).k; };
  // The bulk of a row, away from its few largest elements: of the warps' smallest maximum of a thread the largest.
  const bool some = tid * 4 < p.K;   // this thread has elements of every row
  auto reduce_row = [&](int m, uint32_t mx, float ss) {
    const uint32_t low = __reduce_min_sync(0xffffffffu, some ? mx : 0xffffffffu);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (p.norm_w != nullptr)
      ss = warp_sum(ss);
    if (lane == 0) {
      red[m * W + warp] = mx;
      redf[m * W + warp] = ss;
      redb[m * W + warp] = low == 0xffffffffu ? 0u : low;
    }
  };
  auto finish_rows = [&]() {
    if (tid == 0)
      s_wide = 0;
    __syncthreads();
    for (int m = warp; m < p.M; m += W) {   // a warp per row
      const uint32_t mx = __reduce_max_sync(0xffffffffu, lane < W ? red[m * W + lane] : 0u);
      const uint32_t bulk = __reduce_max_sync(0xffffffffu, lane < W ? redb[m * W + lane] : 0u);
      const float ss = p.norm_w != nullptr ? warp_sum(lane < W ? redf[m * W + lane] : 0.f) : 0.f;
      if (lane == 0) {
        float inv;
        const float scale = fixed_scale(mx, &inv);
        s_scale[m] = scale;
        if (mx != 0u && mx < 0x7f800000u && __uint_as_float(bulk) * scale < 2097152.f)   // 2^21 units: 2^-22 is as f32 sums round
          s_wide = 1;
        s_inv[m] = p.norm_w != nullptr ? inv * rsqrtf(ss * (1.0f / (float)p.K) + p.eps) : inv;
      }
    }
    __syncthreads();
  };
  auto add4 = [&](float4 v, float &ss) {
    ss = fmaf(v.x, v.x, ss);
    ss = fmaf(v.y, v.y, ss);
    ss = fmaf(v.z, v.z, ss);
    ss = fmaf(v.w, v.w, ss);
  };
  auto stage_tail = [&]() {
    if constexpr (U4) {
      const int padded = (nu + 3) & ~3;   // units beyond the row: zero
      for (int m = 0; m < p.M; ++m)
        for (int i = tid; i < ((padded * 8 + 31) & ~31); i += nthr) {
          const int j = i / padded, u = i - j * padded, k = p.tail_k0 + j * nu * 4 + 4 * u;
          const bool in = j < 8 && u < nu;
          const float4 v = in ? normed<XF>(p, k, act4<XF>(p, m, k)) : make_float4(0.f, 0.f, 0.f, 0.f);
          if (j < 8)   // a multiple of four lanes either way
            store_u4_tail<COLS>(tplanes, tstart, u, j, m, v, s_scale[m]);
        }
    }
  };
  bool staged = false;
  constexpr int kR = U4 ? 3 : 6;   // groups a thread keeps in registers: K <= 12288 with 16 warps
  if (XF && p.reg_x) {
    // one row, one read: the values stay in registers between the two passes
    float4 v[kR], v2[U4 ? kR : 1];
    const int groups = p.units * 4;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      const int i = tid + u * nthr;
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (U4)
        v2[u % (U4 ? kR : 1)] = v[u];
      if (i < groups) {
        const int k = k_of(i, p.units);
        v[u] = act4<XF>(p, 0, k);
        if constexpr (U4)
          v2[u] = act4<XF>(p, 0, k + 16);
      }
    }
    uint32_t mx = 0;
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      const int i = tid + u * nthr;
      if (i < groups) {
        const int k = k_of(i, p.units);
        add4(v[u], ss);
        v[u] = normed<XF>(p, k, v[u]);
        mx = max(mx, absbits4(v[u]));
        if constexpr (U4) {
          add4(v2[u], ss);
          v2[u] = normed<XF>(p, k + 16, v2[u]);
          mx = max(mx, absbits4(v2[u]));
        }
      }
    }
    if (U4)
      for (int k = p.tail_k0 + tid * 4; k < p.K; k += nthr * 4) {
        const float4 x = act4<XF>(p, 0, k);
        add4(x, ss);
        mx = max(mx, absbits4(normed<XF>(p, k, x)));
      }
    reduce_row(0, mx, ss);
    finish_rows();
    const float scale = s_scale[0];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      const int i = tid + u * nthr;
      if (i < groups) {
        if constexpr (U4)
          store_u4<COLS>(planes, start, group_u4(i), 0, v[u], v2[u], scale);
        else
          store_i8<COLS>(planes, group_i8(i, p.units), 0, v[u], scale);
      }
    }
    if (U4 && nu > 0)
      stage_tail();
    staged = true;
    __syncthreads();
  } else {
    // four rows at a time, one or two loads of each in flight per thread: a row after the other is a chain of M latencies
    for (int m0 = 0; m0 < p.M; m0 += 4) {
      uint32_t mx[4] = {0, 0, 0, 0};
      float ss[4] = {0.f, 0.f, 0.f, 0.f};
      constexpr int kU = XF ? 2 : 1;   // (16-bit loads bring more code)
      for (int k = tid * 4; k < p.K; k += kU * nthr * 4) {
        float4 v[4][kU];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int u = 0; u < kU; ++u)
            v[q][u] = act4<XF>(p, min(m0 + q, p.M - 1), k + u * nthr * 4);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            if (p.norm_w != nullptr)
              add4(v[q][u], ss[q]);
            mx[q] = max(mx[q], absbits4(normed<XF>(p, k + u * nthr * 4, v[q][u])));
          }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (m0 + q < p.M)
          reduce_row(m0 + q, mx[q], ss[q]);
    }
    finish_rows();
    if (U4 && nu > 0)
      stage_tail();
  }
  // planes of the slab that starts at step s0; all rows' groups as one list, four loads in flight per thread
  auto stage = [&](int s0) {
    const int k0 = s0 * (U4 ? 512 : 256);
    constexpr int kU = U4 ? 1 : COLS > 16 ? 8 : 4;
    const int units = min(p.slab_k / (U4 ? 32 : 16), p.units - k0 / (U4 ? 32 : 16));
    const int groups = units * 4;   // per row (int4: a multiple of 128, so a warp never straddles two rows)
    const int total = groups * p.M;
    const uint32_t magic = 0xffffffffu / (uint32_t)groups + 1;   // i / groups exactly for i < total <= 2^16
    auto row_of = [&](int i) { return groups > 1 ? (int)__umulhi((uint32_t)i, magic) : i; };
    if constexpr (U4) {   // the next group is loaded while this one is stored: one copy of the code, which is long and cold
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f), v2 = v;
      auto load = [&](int i, float4 &x, float4 &y) {
        if (i < total) {
          const int m = row_of(i), k = k0 + k_of(i - m * groups, units);
          x = act4<XF>(p, m, k);
          y = act4<XF>(p, m, k + 16);
        }
      };
      load(tid, v, v2);
#pragma unroll 1
      for (int i = tid; i < total; i += nthr) {
        float4 nv = v, nv2 = v2;
        load(i + nthr, nv, nv2);
        const int m = row_of(i), k = k0 + k_of(i - m * groups, units);
        store_u4<COLS>(planes, start, group_u4(i - m * groups), m, normed<XF>(p, k, v), normed<XF>(p, k + 16, v2), s_scale[m]);
        v = nv;
        v2 = nv2;
      }
    } else {
      for (int i0 = tid; i0 < total; i0 += kU * nthr) {
        float4 v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int i = i0 + u * nthr;
          if (i < total) {
            const int m = row_of(i);
            v[u] = act4<XF>(p, m, k0 + k_of(i - m * groups, units));
          }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int i = i0 + u * nthr;
          if (i < total) {
            const int m = row_of(i), k = k0 + k_of(i - m * groups, units);
            store_i8<COLS>(planes, group_i8(i - m * groups, units), m, normed<XF>(p, k, v[u]), s_scale[m]);
          }
        }
      }
    }
  };

  if (s_wide) {   // (the same in all CTAs)
    float_rows<KIND, GROUPED, XF>(p, s_scale, s_inv);
    return;
  }
  int s = kp, buf = 0;
  for (int r = 0; r < p.rounds; ++r) {
    const int64_t tile = tile_of(r);
    const bool mine = tile < p.tiles;
    // what the epilogue needs is requested before the sums: lane l serves row l % 16
    const int64_t erow = min(tile * kTileRows + (lane & 15), (int64_t)p.N - 1);
    float e_scale = 1.f, e_bias = 0.f, e_res = 0.f;
    if (mine) {
      if (!GROUPED)
        e_scale = load_as_float(p.scale, p.scale_dtype, erow);
      if (p.bias != nullptr)
        e_bias = __ldg(p.bias + erow);
      if (p.residual != nullptr && p.M == 1)
        e_res = p.residual[erow];
    }
    typename std::conditional<U4, AccU4<COLS, GROUPED>, AccI8<COLS>>::type acc;
    acc.clear();
    for (int s0 = 0; s0 < p.steps || s0 == 0; s0 += p.slab_steps) {
      if (!(one_slab && staged)) {
        if (staged)
          __syncthreads();
        stage(s0);
        __syncthreads();
        staged = true;
      }
      if (mine) {
        const int end = min(s0 + p.slab_steps, steps);
        for (; s < end; s += p.ks) {
          uint4 nx[8];
          Scales nsc{};
          int64_t nt = tile;
          int s2 = s + p.ks;
          TileRows nrows = rows;
          if (s2 >= steps) {
            s2 = kp;
            nt = r + 1 < p.rounds ? tile_of(r + 1) : p.tiles;
            if (nt < p.tiles)
              nrows = tile_rows(p.w, p.row_bytes, nt * kTileRows, p.N);
          }
          if (nt < p.tiles)
            fetch(nt, nrows, s2, nx, nsc);
          if constexpr (U4)
            acc.step(w, s - s0, planes, start, sc.s0, sc.s8);
          else
            acc.step(w, s - s0, planes);
          rows = nrows;
          sc = nsc;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            w[i] = nx[i];
        }
      }
    }
    s = kp;
    if (!mine)
      continue;
    if constexpr (U4) {
      if (nu > 0) {
        const TileRows tr = tile_rows(p.w + (int64_t)(p.tail_k0 / 32) * 16, p.row_bytes, tile * kTileRows, p.N);
        const int64_t ra = min(tile * kTileRows + (lane >> 2), (int64_t)p.N - 1);
        const int64_t rb = min(tile * kTileRows + (lane >> 2) + 8, (int64_t)p.N - 1);
        const __half *h = reinterpret_cast<const __half *>(p.scale) + p.tail_k0 / 128;
        acc.tail(tr, kp, p.ks, nu, tplanes, tstart, h + ra * p.ngroups, h + rb * p.ngroups);
      }
    }
    // ---- the tile's sums: planes -> f32, k shares of the warps, epilogue -----------------------------------------
    float *mypart = part + ((size_t)(buf * p.slots + slot) * p.ks + kp) * p.M * kTileRows;
#pragma unroll
    for (int n = 0; n < kTiles<COLS>; ++n) {
      float v0, v1;
      acc.combine(n, v0, v1);
      const int m = 2 * n + ((lane & 3) >> 1);
      if ((lane & 1) == 0 && m < p.M) {
        mypart[m * kTileRows + (lane >> 2)] = v0 * s_inv[m];
        mypart[m * kTileRows + (lane >> 2) + 8] = v1 * s_inv[m];
      }
    }
    if (p.ks > 1)
      asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(p.ks * 32) : "memory");
    else
      __syncwarp();
    const float *sums = part + (size_t)(buf * p.slots + slot) * p.ks * p.M * kTileRows;
    const int per = p.M * kTileRows;
    for (int i = kp * 32 + lane; i < ((per + 31) & ~31); i += p.ks * 32) {
      const int m = i >> 4, rr = i & 15;   // rr == lane % 16
      float v = 0.f;
      if (m < p.M) {
        for (int q = 0; q < p.ks; ++q)
          v += sums[q * per + i];
        if (!GROUPED)
          v *= e_scale;
        if (p.bias != nullptr)
          v = e_bias + v;
      }
      const int64_t row = tile * kTileRows + rr;
      int64_t o = (int64_t)m * p.y_ld + row;
      if (p.silu_pairs) {
        const float up = __shfl_down_sync(0xffffffffu, v, 1);
        if (m >= p.M || (rr & 1) || row + 1 >= p.N)
          continue;
        v = silu_gate(v, up);
        o = (int64_t)m * p.y_ld + (row >> 1);
      } else {
        if (m >= p.M || row >= p.N)
          continue;
        if (p.residual != nullptr)
          v = (p.M == 1 ? e_res : p.residual[o]) + v;
      }
      if (p.y_dtype == B200_F32)
        ((float *)p.y)[o] = p.accumulate ? ((float *)p.y)[o] + v : v;
      else
        ((__half *)p.y)[o] = __float2half_rn(p.accumulate ? __half2float(((__half *)p.y)[o]) + v : v);
    }
    __syncwarp();
    buf ^= 1;
  }
}

int device_sms() {
  static int sms[64];
  static std::once_flag once[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return 148;
  std::call_once(once[dev], [&] { cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev); });
  return sms[dev] > 0 ? sms[dev] : 148;
}

constexpr int kMmaSmem = 224 * 1024;

template <int KIND, int COLS, bool GROUPED, bool XF> static int launch_mma(MmaP &p, cudaStream_t st) {
  auto kern = gemv_mma_kernel<KIND, COLS, GROUPED, XF>;
  constexpr bool U4 = KIND == B200_W_U4;
  constexpr int W = kMaxWarps<COLS>, SB = kSetBytes<COLS>;
  const int sms = device_sms();
  // ---- activation slab: everything, or as many whole blocks as fit ------------------------------------------------
  const int blk = U4 ? 1024 : 512, span = U4 ? p.tail_k0 : p.units * 16;
  const int tsets = (p.tunits + 3) / 4;
  const int tail_bytes = tsets * 4 * SB, tstart_bytes = tsets * 8 * COLS * 4;
  const int part_bytes = 2 * W * p.M * kTileRows * 4, red_bytes = p.M * (3 * W + 2) * 4;
  const int room = kMmaSmem - tail_bytes - tstart_bytes - part_bytes - red_bytes;
  const int per_blk = blk / 64 * SB + (U4 ? 16 * COLS * 4 : 0);   // a set covers 64 k
  int nblk = (span + blk - 1) / blk;
  if ((int64_t)nblk * per_blk > room)
    nblk = room / per_blk;
  if (nblk < 1 && span > 0)
    return fail(B200_ELIMIT, "gemv: no room for one block of activation planes (M=%d)", p.M);
  p.slab_k = nblk * blk;
  p.slab_steps = nblk > 0 ? p.slab_k / (U4 ? 512 : 256) : 1;
  p.start_off = p.slab_k / 64 * SB;
  p.tail_off = p.start_off + (U4 ? p.slab_k / 64 * COLS * 4 : 0);
  p.tstart_off = p.tail_off + tail_bytes;
  p.part_off = p.tstart_off + tstart_bytes;
  p.red_off = p.part_off + part_bytes;
  const int smem = p.red_off + red_bytes;
  // ---- warps per tile: fewest (rounds x steps per round), a round's fixed cost counted as about one step ------------
  p.tiles = (p.N + kTileRows - 1) / kTileRows;
  const int all = p.steps + (p.tunits + kStepUnits - 1) / kStepUnits;
  float best = 0.f;
  p.ks = 0;
  for (int ks : {1, 2, 3, 4, 5, 6, 8, 12, 16}) {
    if (ks > W || (ks > 1 && ks > all))
      continue;
    const int64_t per_round = (int64_t)sms * (W / ks);
    const float cost = (float)((p.tiles + per_round - 1) / per_round) * ((float)((all + ks - 1) / ks) + 0.75f);
    if (p.ks == 0 || cost < best) {
      best = cost;
      p.ks = ks;
    }
  }
  // tiles per CTA and round: no more than it takes to use every SM
  p.slots = W / p.ks;
  const int64_t per_sm = ((int64_t)p.tiles + sms - 1) / sms;
  if (per_sm < p.slots)
    p.slots = (int)per_sm;
  const int64_t ctas = ((int64_t)p.tiles + p.slots - 1) / p.slots;
  const int grid = (int)(ctas < sms ? ctas : sms);
  p.rounds = (int)((ctas + grid - 1) / grid);
  // Several rows: the staging takes longer than a narrow projection's products, and few warps issue it at their latency, so
  // all warps take part (int4 14336 x 4096, 5 rows: 7 warps hold tiles).
  const int threads = (p.M > 1 ? W : p.slots * p.ks) * 32;
  p.reg_x = p.M == 1 && nblk * blk >= span && p.units * 4 <= (U4 ? 3 : 6) * threads;
  static RaisedOn raised;
  if (int rc = raise_shared_limit(raised, (const void *)kern, kMmaSmem))
    return rc;
  kern<<<grid, threads, smem, st>>>(p);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

// One row: short rows over few weights are faster on the CUDA cores (a chain of launch, load, product; no digits to make).  Device
// time per call in a graph, weights from memory, us here / there: int8 K = 512: 4.0 / 3.1 at 1 MB, 4.8 / 4.9 at 5, 6.2 / 7.1 at 10;
// K = 1536: 4.4 / 4.6 at 1, 5.3 / 5.4 at 6, 6.4 / 6.0 at 10 (weights in L2: 4.2 / 3.6 at 2); K = 2560: 5.5 / 6.1 at 1; K = 4096:
// 5.4 / 8.4 at 1, 6.0 / 8.7 at 6; K = 8960: 7.9 / 15.4 at 1; K = 14336: 13.0 / 21.5 at 1.  int4 K = 512: 7.3 / 5.0 at 1 MB, 6.9 / 7.0
// at 2, 8.4 / 14 at 6; K = 1536: 7.5 / 6.9 at 1, 7.2 / 8.1 at 3; K = 2560: 6.6 / 8.7 at 0.5; K = 8960: 9.6 / 23 at 1.  (f32 rows of up to four whole blocks have a
// quicker form there: K = 4096 5.3 / 6.1 at 0.5 MB from memory, 5.2 / 4.8 at 1.2 MB from L2.)
// int4 rows of 2.5 to five blocks of 1024: there, per-channel scales cost nothing and whole blocks of f32 rows have a quicker form; here, a
// part of a block is staged by itself, and the ten steps of five blocks go to five warps, too few to keep the row in registers.  From
// memory, us here / there (in brackets from L2), 1024 rows, f32: per channel K = 2560 6.5 / 4.9 (5.7 / 3.8), 3584 7.3 / 5.8 (6.2 / 4.4), 5120 9.1 /
// 6.8 (8.4 / 5.0), 6144 6.5 / 7.8 (6.0 / 5.5); groups of 128 2560 7.0 / 8.8 (6.2 / 7.7), 3584 7.8 / 11.3 (6.8 / 9.6), 5120 9.6 / 7.2 (9.0 /
// 5.7), 6144 6.6 / 8.3 (6.2 / 6.4); bf16: per channel 3584 10.6 / 8.7 (9.7 / 7.3), 4096 7.8 / 9.3 (7.5 / 7.8), 5120 11.2 / 11.1 (10.6 / 9.3), groups
// 2560 8.9 / 10.8, 5120 11.7 / 12.6.  (int8 rows of 2560 to 3071 that lie in L2 take 0.2 to 0.8 us more here, from memory 0.5 to 1.5 less.)
static bool one_row_is_short(const b200_weight *w, const b200_gemv_args *a) {
  const int64_t bytes = packed_row_bytes(w->kind, w->K) * w->N, mb = 1 << 20;
  if (w->kind == B200_W_I8 || w->K < 2560)
    return w->K < 2560 && bytes < (w->kind == B200_W_I8 ? 6 * mb : 3 * mb);
  const bool whole = w->K % 1024 == 0, grouped = w->group > 0 && w->group < w->K;
  if (w->K > 5120 || (grouped && !whole) || (a->x_dtype != B200_F32 && (grouped || w->K == 4096)))
    return false;
  return bytes < (w->K == 4096 ? 3 * mb : 6 * mb);
}

// Whether the integer-MMA kernel takes this call: per-channel int8 or int4 (any scale type), or int4 in groups of 128
// with f16 scales (the group is then one 4-element column of a packed block), up to K = 65536 (s32 sums).
bool gemv_mma_takes(const b200_weight *w, const b200_gemv_args *a) {
  if (w->K > 65536 || (w->kind != B200_W_I8 && w->kind != B200_W_U4) || (a->M == 1 && one_row_is_short(w, a)))
    return false;
  const bool grouped = w->kind == B200_W_U4 && w->group > 0 && w->group < w->K;
  return !grouped || (w->group == 128 && w->scale_dtype == B200_F16 && w->K % 128 == 0);
}

int gemv_mma_run(const b200_weight *w, const b200_gemv_args *a, cudaStream_t st) {
  MmaP p{};
  p.x = a->x;
  p.w = (const uint8_t *)w->w;
  p.scale = w->scale;
  p.bias = w->bias;
  p.residual = a->residual;
  p.norm_w = a->norm_weight;
  p.y = a->y;
  p.x_ld = a->x_ld ? a->x_ld : w->K;
  p.y_ld = a->y_ld ? a->y_ld : (a->silu_pairs ? w->N / 2 : w->N);
  p.K = (int)w->K;
  p.Kp = (int)packed_k(w->kind, w->K);
  p.row_bytes = packed_row_bytes(w->kind, w->K);
  p.N = (int)w->N;
  p.M = a->M;
  p.x_dtype = a->x_dtype;
  p.y_dtype = a->y_dtype;
  p.scale_dtype = w->scale_dtype;
  p.accumulate = a->accumulate;
  p.silu_pairs = a->silu_pairs;
  p.eps = a->norm_eps;
  const bool u4 = w->kind == B200_W_U4, grouped = u4 && w->group > 0 && w->group < w->K;
  p.tail_k0 = u4 ? p.Kp / 1024 * 1024 : p.Kp;
  p.units = u4 ? p.tail_k0 / 32 : p.Kp / 16;
  p.steps = (p.units + kStepUnits - 1) / kStepUnits;
  p.tunits = (p.Kp - p.tail_k0) / 32 * (u4 ? 1 : 0);
  p.ngroups = grouped ? (int)(w->K / 128) : 1;
  p.scale_vec = p.ngroups % 8 == 0 && (reinterpret_cast<uintptr_t>(w->scale) & 15) == 0;
  p.x_vec = a->x_dtype != B200_F32 && p.x_ld % 4 == 0 && (reinterpret_cast<uintptr_t>(a->x) & 7) == 0;
  const bool xf = a->x_dtype == B200_F32 && p.x_ld % 4 == 0 && w->K % 4 == 0 && (reinterpret_cast<uintptr_t>(a->x) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(a->norm_weight) & 15) == 0;
#define B200_MMA(COLS_)                                                                                                  \
  if (!u4)                                                                                                             \
    return xf ? launch_mma<B200_W_I8, COLS_, false, true>(p, st) : launch_mma<B200_W_I8, COLS_, false, false>(p, st);      \
  if (grouped)                                                                                                         \
    return xf ? launch_mma<B200_W_U4, COLS_, true, true>(p, st) : launch_mma<B200_W_U4, COLS_, true, false>(p, st);        \
  return xf ? launch_mma<B200_W_U4, COLS_, false, true>(p, st) : launch_mma<B200_W_U4, COLS_, false, false>(p, st)
  if (a->M == 1) { B200_MMA(4); }
  if (a->M == 2) { B200_MMA(8); }
  if (a->M <= 4) { B200_MMA(16); }
  if (a->M <= 6) { B200_MMA(24); }
  if (a->M <= 8) { B200_MMA(32); }
  if (a->M <= 12) { B200_MMA(48); }
  B200_MMA(64);
#undef B200_MMA
}

} // namespace b200
