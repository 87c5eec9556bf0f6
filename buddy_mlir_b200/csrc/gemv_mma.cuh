// Weight-only GEMV on the integer tensor cores: the pieces shared by b200_gemv and the persistent decode kernel.
//
// An activation row is turned into four int8 planes of one fixed-point number: with e the exponent of the row's
// largest magnitude, X = rint(x * 2^(29-e)) (|X| < 2^30, the scale is a power of two, so every element within 2^-7 of
// the largest is exact and the rest is within 2^-31 of it: tighter than f32 sums until one channel is some thousand
// times the rest; b200_gemv multiplies such calls in f32), and
// X = p0*2^24 + p1*2^16 + p2*2^8 + p3 with signed bytes.  The planes are columns of the B operand of
// mma.m16n8k32.s8: sixteen weight rows are A, as stored, and the products add up exactly in s32.
//   int8: no conversion at all: 2 loads and 2 MMAs per 1024 weights (the FFMA form: 2 instructions per weight and lane);
//   int4: PRMT + mask, 8 instructions per 16 nibbles; the zero point -8*sum(X) is the accumulator's start value.
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int kTileRows = 16;
constexpr int kStepUnits = 16;   // 16-byte units of a row per step: 256 k of int8, 512 k of int4

__device__ __forceinline__ uint4 ld_weights(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Fixed-point scale of a row from the bit pattern of its largest magnitude, so that |X| < 2^(TOP+1); *inv undoes it.  A row
// with an infinity or a NaN gets inv = NaN, so its results are NaN.
template <int TOP = 29> __device__ __forceinline__ float fixed_scale(uint32_t absbits, float *inv) {
  const int e = max((int)(absbits >> 23) - 127, -90);
  *inv = absbits >= 0x7f800000u ? __uint_as_float(0x7fffffffu) : __uint_as_float((uint32_t)(e - TOP + 127) << 23);
  return __uint_as_float((uint32_t)(TOP - e + 127) << 23);
}
// The four signed digits of X, most significant in the top byte.
__device__ __forceinline__ uint32_t fixed_digits(float v, float scale) {
  return (uint32_t)(__float2int_rn(v * scale) + 0x00808080) ^ 0x00808080u;
}
// Digits of four elements -> one word per plane (plane 0 = most significant), element i in byte i.
__device__ __forceinline__ void plane_words(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&w)[4]) {
  const uint32_t lo01 = __byte_perm(a, b, 0x5140), hi01 = __byte_perm(a, b, 0x7362);
  const uint32_t lo23 = __byte_perm(c, d, 0x5140), hi23 = __byte_perm(c, d, 0x7362);
  w[3] = __byte_perm(lo01, lo23, 0x5410);
  w[2] = __byte_perm(lo01, lo23, 0x7632);
  w[1] = __byte_perm(hi01, hi23, 0x5410);
  w[0] = __byte_perm(hi01, hi23, 0x7632);
}

// ---- planes in shared memory, in the order the MMA lanes read them -----------------------------------------------
// int8: set i = four units 4i..4i+3 of the packed row; chunk (set, column, t) of 16 bytes = the column's words for the
// four 4-element groups of unit 4i+t.  int4 (whole 1024-element blocks): set (block, p, wi), chunk = {b0, b1} of groups
// 2wi and 2wi+1 over units 8p+t and 8p+4+t.  COLS columns, 4*m + plane: 4 for a single row (the MMA's other four columns
// then repeat them), else the MMA's multiples of 8; columns nobody wrote only reach sums nobody reads.  64 bytes
// between the sets spread the stores of a warp over the banks; all offsets inside a step are compile-time constants.
template <int COLS> constexpr int kSetBytes = COLS * 64 + 64;
template <int COLS> constexpr int kTiles = COLS < 8 ? 1 : COLS / 8;   // MMA column tiles
template <int COLS> __device__ __forceinline__ int plane_at(int set, int m, int plane, int t) {
  return set * kSetBytes<COLS> + ((4 * m + plane) * 4 + t) * 16;
}
template <int COLS> __device__ __forceinline__ int lane_at() {   // this lane's chunk of set 0, column tile 0
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  return ((COLS < 8 ? g & 3 : g) * 4 + t) * 16;
}

// Group idx of a row slab (int8): four consecutive k.  Returns its first k relative to the slab; `units` = units in the slab.
struct GroupI8 {
  int set, t, j, k;
};
__device__ __forceinline__ GroupI8 group_i8(int idx, int units) {
  const int b = idx >> 7, r = idx & 127;
  const int nu = min(32, units - b * 32);
  GroupI8 g;
  const int l = r >> 2;
  g.j = r & 3;
  g.set = b * 8 + (l >> 2);
  g.t = l & 3;
  g.k = b * 512 + g.j * (nu * 4) + 4 * l;
  return g;
}
template <int COLS>
__device__ __forceinline__ void store_i8(uint8_t *planes, const GroupI8 &g, int m, float4 v, float scale) {
  uint32_t w[4];
  plane_words(fixed_digits(v.x, scale), fixed_digits(v.y, scale), fixed_digits(v.z, scale), fixed_digits(v.w, scale), w);
#pragma unroll
  for (int pl = 0; pl < 4; ++pl)
    *reinterpret_cast<uint32_t *>(planes + plane_at<COLS>(g.set, m, pl, g.t) + g.j * 4) = w[pl];
}
// Group idx of a slab (int4): k .. k+3 and k+16 .. k+19 of group j.
struct GroupU4 {
  int b, j, p, t, k;
};
__device__ __forceinline__ GroupU4 group_u4(int idx) {
  GroupU4 g;
  g.b = idx >> 7;
  g.j = (idx >> 4) & 7;
  g.p = (idx >> 2) & 3;
  g.t = idx & 3;
  g.k = g.b * 1024 + g.j * 128 + 4 * (8 * g.p + g.t);
  return g;
}
// Accumulator start values of the int4 sums, -8 * (sum of the plane over the group's k in this step): [step][wi][column
// pair][group parity][column parity], so that a lane reads both groups of a word with one 16-byte load.  The float bias
// 1.5 * 2^23 is part of them: the s32 sum then IS the bit pattern of 1.5 * 2^23 + sum (|sum| < 2^22), and leaves the
// integer domain with one FADD (I2F runs at an eighth of that rate).
constexpr int kFloatBias = 0x4B400000;
template <int COLS> __device__ __forceinline__ int start_u4(int step, int wi, int col, int jj) {
  return (step * 4 + wi) * (COLS * 2) + (col >> 1) * 4 + jj * 2 + (col & 1);
}
// The whole warp takes part (consecutive idx, so eight neighbouring lanes share a half block's group).
template <int COLS>
__device__ __forceinline__ void store_u4(uint8_t *planes, int *start, const GroupU4 &g, int m, float4 v, float4 u,
                                         float scale) {
  uint32_t w0[4], w1[4];
  plane_words(fixed_digits(v.x, scale), fixed_digits(v.z, scale), fixed_digits(u.x, scale), fixed_digits(u.z, scale), w0);
  plane_words(fixed_digits(v.y, scale), fixed_digits(v.w, scale), fixed_digits(u.y, scale), fixed_digits(u.w, scale), w1);
  const int set = (g.b * 4 + g.p) * 4 + (g.j >> 1);
#pragma unroll
  for (int pl = 0; pl < 4; ++pl) {
    *reinterpret_cast<uint2 *>(planes + plane_at<COLS>(set, m, pl, g.t) + (g.j & 1) * 8) =
        make_uint2(w0[pl], w1[pl]);
    int s = __dp4a((int)w0[pl], 0x01010101, __dp4a((int)w1[pl], 0x01010101, 0));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    if ((g.t | (g.p & 1)) == 0)
      start[start_u4<COLS>(g.b * 2 + (g.p >> 1), g.j >> 1, 4 * m + pl, g.j & 1)] = kFloatBias - 8 * s;
  }
}
// The last K % 1024 elements of an int4 row: a short block of nu = n / 32 units, group j covering k = j*(n/8) + 4*unit.
// A scale group of 128 may end inside group j, but only at a multiple of four units, so these are multiplied four units
// at a time (the other half of the MMA's k is zero).  Chunk (set = four units, wi), start value per (set, wi).
template <int COLS>
__device__ __forceinline__ void store_u4_tail(uint8_t *planes, int *start, int unit, int j, int m, float4 v, float scale) {
  uint32_t w0[4], w1[4];
  plane_words(fixed_digits(v.x, scale), fixed_digits(v.z, scale), 0, 0, w0);
  plane_words(fixed_digits(v.y, scale), fixed_digits(v.w, scale), 0, 0, w1);
  const int set = (unit >> 2) * 4 + (j >> 1);
#pragma unroll
  for (int pl = 0; pl < 4; ++pl) {
    *reinterpret_cast<uint2 *>(planes + plane_at<COLS>(set, m, pl, unit & 3) + (j & 1) * 8) =
        make_uint2(w0[pl], w1[pl]);
    int s = __dp4a((int)w0[pl], 0x01010101, __dp4a((int)w1[pl], 0x01010101, 0));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((unit & 3) == 0)
      start[start_u4<COLS>(unit >> 2, j >> 1, 4 * m + pl, j & 1)] = kFloatBias - 8 * s;
  }
}

// ---- the row tile of one warp -------------------------------------------------------------------------------------
// Weights of one step: units 16s + 4q + t of rows g (w[2q]) and g + 8 (w[2q+1]) of the tile.  Lane = 4g + t.
struct TileRows {
  const uint8_t *r0, *r8;   // row pointers, + 16*t applied
};
__device__ __forceinline__ TileRows tile_rows(const uint8_t *w, int64_t row_bytes, int64_t row0, int64_t N) {
  const int lane = threadIdx.x & 31;
  const int64_t a = min(row0 + (lane >> 2), N - 1), b = min(row0 + (lane >> 2) + 8, N - 1);   // clamped rows are not stored
  return {w + a * row_bytes + (lane & 3) * 16, w + b * row_bytes + (lane & 3) * 16};
}
__device__ __forceinline__ void load_step(const TileRows &r, int s, int units, uint4 (&w)[8]) {
  const int u0 = s * kStepUnits + (threadIdx.x & 3);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const bool in = u0 + 4 * q < units;   // beyond the row: zero weights
    const int64_t off = (int64_t)(s * kStepUnits + 4 * q) * 16;
    w[2 * q] = in ? ld_weights(r.r0 + off) : make_uint4(0, 0, 0, 0);
    w[2 * q + 1] = in ? ld_weights(r.r8 + off) : make_uint4(0, 0, 0, 0);
  }
}

template <int COLS> struct AccI8 {
  static constexpr int NT = kTiles<COLS>;
  int c[NT][4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int n = 0; n < NT; ++n)
      c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0;
  }
  // s: step relative to the slab whose planes are staged
  __device__ __forceinline__ void step(const uint4 (&w)[8], int s, const uint8_t *planes) {
    const uint8_t *at = planes + lane_at<COLS>() + s * (4 * kSetBytes<COLS>);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const uint4 b = *reinterpret_cast<const uint4 *>(at + q * kSetBytes<COLS> + n * 512);
        mma_s8(c[n], w[2 * q].x, w[2 * q + 1].x, w[2 * q].y, w[2 * q + 1].y, b.x, b.y);
        mma_s8(c[n], w[2 * q].z, w[2 * q + 1].z, w[2 * q].w, w[2 * q + 1].w, b.z, b.w);
      }
  }
  // Plane sums -> this lane pair's rows g (v0) and g + 8 (v1) of activation row m = 2n + t/2, in units of the row's inv.
  __device__ __forceinline__ void combine(int n, float &v0, float &v1) const {
    const bool lowp = threadIdx.x & 1;   // odd t: planes 2 and 3
    const float f0 = lowp ? 256.f : 16777216.f, f1 = lowp ? 1.f : 65536.f;
    v0 = fmaf((float)c[n][0], f0, (float)c[n][1] * f1);
    v1 = fmaf((float)c[n][2], f0, (float)c[n][3] * f1);
    v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
    v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
  }
};

// GROUPED: one f16 scale per 128 k; the group sums are exact integers, scaled and added in f32.  Otherwise plain sums.
template <int COLS, bool GROUPED> struct AccU4 {
  static constexpr int NT = kTiles<COLS>;
  float f[GROUPED ? NT : 1][4];
  int c[GROUPED ? 1 : NT][4];
  __device__ __forceinline__ void clear() {
    if constexpr (GROUPED) {
#pragma unroll
      for (int n = 0; n < NT; ++n)
        f[n][0] = f[n][1] = f[n][2] = f[n][3] = 0.f;
    } else {
#pragma unroll
      for (int n = 0; n < NT; ++n)
        c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0;
    }
  }
  template <int JJ> __device__ __forceinline__ void begin(int (&d)[JJ][NT][4], const int *start, int step, int wi, int j0) {
    const int t = COLS < 8 ? threadIdx.x & 1 : threadIdx.x & 3;   // the lane's accumulator columns are 2t and 2t + 1
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int *at = start + start_u4<COLS>(step, wi, 2 * t, 0) + n * 16 + j0 * 2;
      int4 z = make_int4(0, 0, 0, 0);
      if constexpr (JJ == 2)
        z = *reinterpret_cast<const int4 *>(at);
      else
        *reinterpret_cast<int2 *>(&z) = *reinterpret_cast<const int2 *>(at);
      d[0][n][0] = d[0][n][2] = z.x;
      d[0][n][1] = d[0][n][3] = z.y;
      if constexpr (JJ == 2) {
        d[1][n][0] = d[1][n][2] = z.z;
        d[1][n][1] = d[1][n][3] = z.w;
      }
    }
  }
  // one group's sums into the row sums; k0 / k8: the group's scale for rows g and g + 8
  __device__ __forceinline__ void finish(const int (&d)[NT][4], float k0, float k8) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      if constexpr (GROUPED) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          f[n][i] = fmaf(__int_as_float(d[n][i]) - 12582912.0f, i < 2 ? k0 : k8, f[n][i]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          c[n][i] += d[n][i] - kFloatBias;
      }
    }
  }
  // s: step (half block) relative to the slab; sc0 / sc8: the eight f16 group scales of the block for rows g and g + 8
  __device__ __forceinline__ void step(const uint4 (&w)[8], int s, const uint8_t *planes, const int *start,
                                       const uint4 &sc0, const uint4 &sc8) {
    const uint8_t *lane = planes + lane_at<COLS>() + s * (8 * kSetBytes<COLS>);
    constexpr int JJ = NT <= 3 ? 2 : 1;   // groups in work at a time, as registers allow (5 rows 14336 x 4096: 29.1 us with 1, 27.0 with 2)
#pragma unroll
    for (int wi = 0; wi < 4; ++wi)
#pragma unroll
      for (int j0 = 0; j0 < 2; j0 += JJ) {
        int d[JJ][NT][4];
        begin<JJ>(d, start, s, wi, j0);
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          const uint32_t ua = word(w[4 * pp], wi), ub = word(w[4 * pp + 2], wi);         // row g: units u, u + 4
          const uint32_t va = word(w[4 * pp + 1], wi), vb = word(w[4 * pp + 3], wi);     // row g + 8
          uint4 b[NT];
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const uint8_t *at = lane + (pp * 4 + wi) * kSetBytes<COLS> + n * 512 + j0 * 8;
            if constexpr (JJ == 2)
              b[n] = *reinterpret_cast<const uint4 *>(at);
            else
              *reinterpret_cast<uint2 *>(&b[n]) = *reinterpret_cast<const uint2 *>(at);
          }
#pragma unroll
          for (int jj = 0; jj < JJ; ++jj) {
            const uint32_t sel = j0 + jj ? 0x7632 : 0x5410;
            const uint32_t x = __byte_perm(ua, ub, sel), y = __byte_perm(va, vb, sel);
            const uint32_t x0 = x & 0x0F0F0F0Fu, x1 = (x >> 4) & 0x0F0F0F0Fu;
            const uint32_t y0 = y & 0x0F0F0F0Fu, y1 = (y >> 4) & 0x0F0F0F0Fu;
#pragma unroll
            for (int n = 0; n < NT; ++n)
              mma_s8(d[jj][n], x0, y0, x1, y1, jj ? b[n].z : b[n].x, jj ? b[n].w : b[n].y);
          }
        }
#pragma unroll
        for (int jj = 0; jj < JJ; ++jj)
          finish(d[jj], half_of(word(sc0, wi), j0 + jj), half_of(word(sc8, wi), j0 + jj));
      }
  }
  // Every step-th set of four units of the short last block (nu units at r); sc0 / sc8: the rows' scales from the block's
  // first group on.
  __device__ __forceinline__ void tail(const TileRows &r, int first, int step, int nu, const uint8_t *planes,
                                       const int *start, const __half *sc0, const __half *sc8) {
    const int t = threadIdx.x & 3;
#pragma unroll 1
    for (int set = first; 4 * set < nu; set += step) {
      const bool in = 4 * set + t < nu;
      const uint4 wa = in ? ld_weights(r.r0 + set * 64) : make_uint4(0, 0, 0, 0);
      const uint4 wb = in ? ld_weights(r.r8 + set * 64) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        int d[1][NT][4];
        begin<1>(d, start, set, j >> 1, j & 1);
        const uint32_t x = word(wa, j >> 1) >> ((j & 1) * 16), y = word(wb, j >> 1) >> ((j & 1) * 16);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint2 b = *reinterpret_cast<const uint2 *>(planes + lane_at<COLS>() + (set * 4 + (j >> 1)) * kSetBytes<COLS> +
                                                           n * 512 + (j & 1) * 8);
          mma_s8(d[0][n], x & 0x0F0Fu, y & 0x0F0Fu, (x >> 4) & 0x0F0Fu, (y >> 4) & 0x0F0Fu, b.x, b.y);
        }
        const int grp = (j * nu * 4 + 16 * set) >> 7;
        finish(d[0], GROUPED ? __half2float(__ldg(sc0 + grp)) : 1.f, GROUPED ? __half2float(__ldg(sc8 + grp)) : 1.f);
      }
    }
  }
  static __device__ __forceinline__ float half_of(uint32_t v, int hi) {
    return __half2float(__ushort_as_half((unsigned short)(hi ? v >> 16 : v & 0xFFFFu)));
  }
  __device__ __forceinline__ void combine(int n, float &v0, float &v1) const {
    const bool lowp = threadIdx.x & 1;
    const float f0 = lowp ? 256.f : 16777216.f, f1 = lowp ? 1.f : 65536.f;
    float a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (GROUPED)
        a[i] = f[n][i];
      else
        a[i] = (float)c[n][i];
    }
    v0 = fmaf(a[0], f0, a[1] * f1);
    v1 = fmaf(a[2], f0, a[3] * f1);
    v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
    v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
  }
  static __device__ __forceinline__ uint32_t word(const uint4 &v, int i) {
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
  }
};

__device__ __forceinline__ float silu_gate(float g, float u) {
  // subgraph0_decode_simplify.mlir:226-231: (g * sigmoid(g)) * u
  const float s = 1.0f / (1.0f + expf(-g));
  return (g * s) * u;
}

} // namespace b200
