// Prefill (many rows at once): the small ops around the dense GEMMs.
//
// buddy-mlir's prefill graph is the decode graph over all max_len rows with a
// causal mask (tools/buddy-codegen/compile_pipeline.py:207-220); its attention
// is flash_attention_for_cpu_prefill_op (frontend/Python/ops/tosa.py:4326-4700:
// blocks of 16 queries x 64 keys, online softmax seeded (-1e30, 0, 0), f32
// inside).  Here row m sits at position pos0 + m and attends to cache rows
// [0, pos0 + m]: the same recurrence over the same keys (masked keys contribute
// exactly 0 in the reference), with the work laid out for a GPU.
#include "common.cuh"

namespace b200 {

namespace {

constexpr float kSeed = -1.0e30f;

// subgraph0_decode_simplify.mlir:46-49, for M tokens
__global__ void embed_rows_kernel(const float *table, const int32_t *tokens, float *x, int64_t H) {
  kernel_go();
  const float4 *src = reinterpret_cast<const float4 *>(table + (int64_t)tokens[blockIdx.x] * H);
  float4 *dst = reinterpret_cast<float4 *>(x + (int64_t)blockIdx.x * H);
  for (int i = threadIdx.x; i < H / 4; i += blockDim.x)
    dst[i] = src[i];
}

// RoPE (and QK-norm) on the q and k heads of every row, K/V rows written to the
// cache: subgraph0_decode_simplify.mlir:52-59, 86-142.  One CTA per row: the angles' cosines and
// sines are made once, a warp takes a head at a time (1000 rows, 14 heads of 128, a layer: 13 us
// for a CTA and the angles per row and head, 5 here).  Where the row's K and V go: row pos0 + m of the
// contiguous cache [kv_heads][max_len][D], or (PAGED) the page of the position, in a pool
// [n_pages][kv_heads][page][D].
constexpr int kRopeThreads = 512;
struct RopeRows {
  float *qkv;
  int64_t ld;
  float *k_cache, *v_cache;   // or pools
  const float *inv_freq, *q_norm, *k_norm;
  float eps;
  int q_heads, kv_heads, D;
  int max_len, pos0;
  int page;                   // PAGED
  const int32_t *row_seq, *row_pos, *block_table;
  int table_stride;
};
// V: neighbouring elements of a lane
template <int V> struct RopeVec {
  float v[V];
  __device__ __forceinline__ void load(const float *p) {
    if constexpr (V == 2) {
      const float2 a = *reinterpret_cast<const float2 *>(p);
      v[0] = a.x;
      v[1] = a.y;
    } else {
      v[0] = *p;
    }
  }
  __device__ __forceinline__ void store(float *p) const {
    if constexpr (V == 2)
      *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    else
      *p = v[0];
  }
};
template <bool PAGED, int V> __global__ void __launch_bounds__(kRopeThreads) rope_rows_kernel(const RopeRows p) {
  extern __shared__ float s_angle[];   // [D / 2] cosines, then sines
  kernel_go();
  const int half = p.D / 2, D = p.D, m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // what the kernel before does not write: the angles, the page
  const int pos = PAGED ? p.row_pos[m] : p.pos0 + m;
  for (int j = threadIdx.x; j < half; j += kRopeThreads) {
    const float th = __fmul_rn(p.inv_freq[j], (float)pos);
    s_angle[j] = cosf(th);
    s_angle[half + j] = sinf(th);
  }
  // of kv head h: row0 + h * step
  const int64_t step = PAGED ? p.page : p.max_len;
  const int64_t row0 = PAGED ? (int64_t)p.block_table[(int64_t)p.row_seq[m] * p.table_stride + pos / p.page] * p.kv_heads * p.page + pos % p.page
                             : pos;
  __syncthreads();
  kernel_wait();
  float *row = p.qkv + (int64_t)m * p.ld;
  for (int head = warp; head < p.q_heads + 2 * p.kv_heads; head += kRopeThreads / 32) {
    float *x = row + (int64_t)head * D;
    const int h = head - p.q_heads;
    RopeVec<V> a, b;
    if (h >= p.kv_heads) {   // v
      float *v = p.v_cache + (row0 + (h - p.kv_heads) * step) * D;
      for (int j = lane * V; j < half; j += 32 * V) {
        a.load(x + j);
        b.load(x + half + j);
        a.store(v + j);
        b.store(v + half + j);
      }
      continue;
    }
    const float *nw = h < 0 ? p.q_norm : p.k_norm;
    float r = 0.f;
    if (nw != nullptr) {
      float ss = 0.f;
      for (int j = lane * V; j < half; j += 32 * V) {
        a.load(x + j);
        b.load(x + half + j);
#pragma unroll
        for (int e = 0; e < V; ++e)
          ss += __fadd_rn(__fmul_rn(a.v[e], a.v[e]), __fmul_rn(b.v[e], b.v[e]));
      }
      r = rsqrtf(__fadd_rn(__fmul_rn(warp_sum(ss), 1.0f / (float)D), p.eps));
    }
    float *k = h < 0 ? nullptr : p.k_cache + (row0 + h * step) * D;
    for (int j = lane * V; j < half; j += 32 * V) {
      a.load(x + j);
      b.load(x + half + j);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        if (nw != nullptr) {
          a.v[e] = __fmul_rn(nw[j + e], __fmul_rn(a.v[e], r));
          b.v[e] = __fmul_rn(nw[j + half + e], __fmul_rn(b.v[e], r));
        }
        const float c = s_angle[j + e], s = s_angle[half + j + e], u = a.v[e], w = b.v[e];
        a.v[e] = __fadd_rn(__fmul_rn(u, c), __fmul_rn(-w, s));
        b.v[e] = __fadd_rn(__fmul_rn(w, c), __fmul_rn(u, s));
      }
      a.store(x + j);
      b.store(x + half + j);
      if (k != nullptr) {
        a.store(k + j);
        b.store(k + half + j);
      }
    }
  }
}
template <bool PAGED> int rope_rows_launch(const RopeRows &p, int M, cudaStream_t st) {
  const bool pairs = p.D % 128 == 0 && (p.ld & 1) == 0 && (((uintptr_t)p.qkv | (uintptr_t)p.k_cache | (uintptr_t)p.v_cache) & 7) == 0;
  return pairs ? launch_after(rope_rows_kernel<PAGED, 2>, dim3(M), kRopeThreads, p.D * 4, st, p)
               : launch_after(rope_rows_kernel<PAGED, 1>, dim3(M), kRopeThreads, p.D * 4, st, p);
}

// Causal attention of M query rows over the cache: grid (M, kv_heads), 4 warps.
// The CTA serves the G query heads that share its kv head (each K/V row is
// loaded once for all of them); a warp owns every 4th key row, lanes own
// D/32 consecutive dims; the four warp states are folded in warp order.
template <int G, int VEC>
__global__ void __launch_bounds__(128)
gqa_prefill_kernel(const float *qkv, int64_t ld, const float *kc, const float *vc, float *out, int64_t ldo,
                   int q_heads, int max_len, int pos0) {
  constexpr int D = VEC * 32, W = 4;
  const int m = blockIdx.x, hk = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int len = min(pos0 + m, max_len - 1) + 1;
  const float scale = rsqrtf((float)D);
  const float *qrow = qkv + (int64_t)m * ld + (int64_t)hk * G * D;
  float qr[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      qr[g][e] = qrow[g * D + lane * VEC + e];
  float mx[G], l[G], acc[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    mx[g] = kSeed;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      acc[g][e] = 0.f;
  }
  const float *kbase = kc + (int64_t)hk * max_len * D + lane * VEC;
  const float *vbase = vc + (int64_t)hk * max_len * D + lane * VEC;
  for (int j = warp; j < len; j += W) {
    float kr[VEC], vr[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      kr[e] = kbase[(int64_t)j * D + e];
      vr[e] = vbase[(int64_t)j * D + e];
    }
    float s[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float d = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        d = fmaf(qr[g][e], kr[e], d);
      s[g] = d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int g = 0; g < G; ++g)
        s[g] += __shfl_xor_sync(0xffffffffu, s[g], o);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      // tosa.py:14245-14252: new_m = max(m, s); alpha = exp(m - new_m); p = exp(s - new_m)
      s[g] *= scale;
      const float nm = fmaxf(mx[g], s[g]);
      const float alpha = expf(mx[g] - nm);
      const float pw = expf(s[g] - nm);
      l[g] = fmaf(l[g], alpha, pw);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        acc[g][e] = fmaf(acc[g][e], alpha, pw * vr[e]);
      mx[g] = nm;
    }
  }
  __shared__ float s_m[W][G], s_l[W][G];
  __shared__ float s_acc[W][G][D];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) {
      s_m[warp][g] = mx[g];
      s_l[warp][g] = l[g];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      s_acc[warp][g][lane * VEC + e] = acc[g][e];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
    const int g = idx / D, d = idx - g * D;
    float M = kSeed;
#pragma unroll
    for (int w = 0; w < W; ++w)
      M = fmaxf(M, s_m[w][g]);
    float L = 0.f, A = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float b = expf(s_m[w][g] - M);
      L = fmaf(s_l[w][g], b, L);
      A = fmaf(s_acc[w][g][d], b, A);
    }
    out[(int64_t)m * ldo + (int64_t)(hk * G + g) * D + d] = __fdiv_rn(A, L);
  }
}

template <int G>
int launch_prefill_attn(const float *qkv, int64_t ld, const float *kc, const float *vc, float *out, int64_t ldo,
                        int q_heads, int kv_heads, int D, int max_len, int pos0, int M, cudaStream_t st) {
  dim3 grid(M, kv_heads);
  if (D == 128)
    gqa_prefill_kernel<G, 4><<<grid, 128, 0, st>>>(qkv, ld, kc, vc, out, ldo, q_heads, max_len, pos0);
  else
    gqa_prefill_kernel<G, 2><<<grid, 128, 0, st>>>(qkv, ld, kc, vc, out, ldo, q_heads, max_len, pos0);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

// ---- paged cache: rows of many sequences, K/V in fixed-size pages -------------------
// Page pool of one cache buffer: [n_pages][kv_heads][page][D] f32.  Row r of the batch
// belongs to sequence row_seq[r] at position row_pos[r]; block_table[seq][pos / page] is
// the page that holds the position.  (buddy-mlir has no paged cache; per sequence the
// arithmetic is that of the contiguous cache above.)

template <int G, int VEC>
__global__ void __launch_bounds__(128)
gqa_paged_kernel(const float *qkv, int64_t ld, const float *k_pool, const float *v_pool, float *out, int64_t ldo,
                 int kv_heads, int page, const int32_t *row_seq, const int32_t *row_pos, const int32_t *block_table,
                 int table_stride) {
  constexpr int D = VEC * 32, W = 4;
  const int m = blockIdx.x, hk = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int len = row_pos[m] + 1;
  const int32_t *table = block_table + (int64_t)row_seq[m] * table_stride;
  const float scale = rsqrtf((float)D);
  const float *qrow = qkv + (int64_t)m * ld + (int64_t)hk * G * D;
  float qr[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      qr[g][e] = qrow[g * D + lane * VEC + e];
  float mx[G], l[G], acc[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    mx[g] = kSeed;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      acc[g][e] = 0.f;
  }
  for (int j = warp; j < len; j += W) {
    const int pg = table[j / page];
    const int64_t crow = (((int64_t)pg * kv_heads + hk) * page + j % page) * D + lane * VEC;
    float kr[VEC], vr[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      kr[e] = k_pool[crow + e];
      vr[e] = v_pool[crow + e];
    }
    float s[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float d = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        d = fmaf(qr[g][e], kr[e], d);
      s[g] = d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int g = 0; g < G; ++g)
        s[g] += __shfl_xor_sync(0xffffffffu, s[g], o);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      s[g] *= scale;
      const float nm = fmaxf(mx[g], s[g]);
      const float alpha = expf(mx[g] - nm);
      const float pw = expf(s[g] - nm);
      l[g] = fmaf(l[g], alpha, pw);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        acc[g][e] = fmaf(acc[g][e], alpha, pw * vr[e]);
      mx[g] = nm;
    }
  }
  __shared__ float s_m[W][G], s_l[W][G];
  __shared__ float s_acc[W][G][D];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) {
      s_m[warp][g] = mx[g];
      s_l[warp][g] = l[g];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      s_acc[warp][g][lane * VEC + e] = acc[g][e];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
    const int g = idx / D, d = idx - g * D;
    float M = kSeed;
#pragma unroll
    for (int w = 0; w < W; ++w)
      M = fmaxf(M, s_m[w][g]);
    float L = 0.f, A = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float b = expf(s_m[w][g] - M);
      L = fmaf(s_l[w][g], b, L);
      A = fmaf(s_acc[w][g][d], b, A);
    }
    out[(int64_t)m * ldo + (int64_t)(hk * G + g) * D + d] = __fdiv_rn(A, L);
  }
}

template <int G>
int launch_paged_attn(const float *qkv, int64_t ld, const float *kp, const float *vp, float *out, int64_t ldo,
                      int kv_heads, int D, int page, const int32_t *row_seq, const int32_t *row_pos,
                      const int32_t *block_table, int table_stride, int M, cudaStream_t st) {
  dim3 grid(M, kv_heads);
  if (D == 128)
    gqa_paged_kernel<G, 4><<<grid, 128, 0, st>>>(qkv, ld, kp, vp, out, ldo, kv_heads, page, row_seq, row_pos,
                                                 block_table, table_stride);
  else
    gqa_paged_kernel<G, 2><<<grid, 128, 0, st>>>(qkv, ld, kp, vp, out, ldo, kv_heads, page, row_seq, row_pos,
                                                 block_table, table_stride);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

// The same scan with the keys of a row cut into chunks of `chunk` positions (paged_chunk(): an eighth of the longest
// context, 32..256), one CTA per (row, kv head, chunk), a warp per 32 keys with 8 rows of V (and 8
// 16-byte pieces of each lane's K row) in flight: the scan is a chain of memory latencies.  Serves decode steps whose
// ranges of keys would be long for a cluster per row (ranges_pay() in paged_decode.cu has the times of both: 2 rows of 8000
// keys, 12 heads on 2, 30 us a layer behind RoPE), and chunks of a prompt that the tensor-core attention does not take.
// Partials (m, l, acc[D]) per query head go to `part`; the CTA that finishes a row's last
// chunk folds them in chunk order.
__host__ __device__ inline int paged_chunk(int max_context) {
  const int c = ((max_context + 7) / 8 + 31) / 32 * 32;
  return c < 32 ? 32 : (c > 256 ? 256 : c);
}
template <int G, int VEC>
__global__ void __launch_bounds__(256, 2)
gqa_paged_split_kernel(const float *qkv, int64_t ld, const float *k_pool, const float *v_pool, float *part,
                       int kv_heads, int page, const int32_t *row_seq, const int32_t *row_pos,
                       const int32_t *block_table, int table_stride, int chunk, int *counters, float *out,
                       int64_t ldo) {
  constexpr int D = VEC * 32, WMAX = 8, VB = 32 / VEC;
  const int W = blockDim.x >> 5;
  kernel_go();
  const int m = blockIdx.x, hk = blockIdx.y, sp = blockIdx.z;
  const int len = row_pos[m] + 1;
  const int j0 = sp * chunk;
  if (j0 >= len)
    return;
  const int j1 = min(len, j0 + chunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t *table = block_table + (int64_t)row_seq[m] * table_stride;
  const float scale = rsqrtf((float)D);
  // the G query vectors of this kv head, shared by every lane (broadcast reads)
  __shared__ __align__(16) float s_q[G][D];
  // row of a key inside the pool, in rows of D floats; positions and pages do not depend on the kernel before
  auto pool_row = [&](int j) { return (table[j / page] * kv_heads + hk) * page + j % page; };
  int ridx = j0 + warp * 32 + lane < j1 ? pool_row(j0 + warp * 32 + lane) : 0;
  kernel_wait();
  const float *qrow = qkv + (int64_t)m * ld + (int64_t)hk * G * D;
  for (int i = threadIdx.x; i < G * D; i += blockDim.x)
    s_q[i / D][i % D] = qrow[i];
  __syncthreads();
  float mx[G], l[G], acc[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    mx[g] = kSeed;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      acc[g][e] = 0.f;
  }
  // A warp takes 32 keys at a time.  Scores: a lane owns one key and walks its K row (no
  // cross-lane reduction per key); softmax over the 32 keys with two warp reductions per query
  // head; values: a lane owns VEC dims, the 32 weights of a head arrive by shuffle.
  for (int jb = j0 + warp * 32; jb < j1; jb += W * 32) {
    const int j = jb + lane;
    const bool live = j < j1;
    if (jb != j0 + warp * 32)
      ridx = live ? pool_row(j) : 0;
    const float *kp = k_pool + (int64_t)ridx * D;
    float sc[G];
#pragma unroll
    for (int g = 0; g < G; ++g)
      sc[g] = 0.f;
    const int nk = min(32, j1 - jb);
    // values of keys t0 .. t0 + VB - 1 of the 32 (beyond nk: the last key again, with weight 0): VB rows in flight
    float vr[VB][VEC];
    auto fetch = [&](int t0) {
#pragma unroll
      for (int u = 0; u < VB; ++u) {
        const float *vp = v_pool + (int64_t)__shfl_sync(0xffffffffu, ridx, min(t0 + u, nk - 1)) * D + lane * VEC;
        if (VEC == 4) {
          const float4 b = *reinterpret_cast<const float4 *>(vp);
          vr[u][0] = b.x; vr[u][1] = b.y; vr[u][2 % VEC] = b.z; vr[u][3 % VEC] = b.w;
        } else {
          const float2 b = *reinterpret_cast<const float2 *>(vp);
          vr[u][0] = b.x; vr[u][1] = b.y;
        }
      }
    };
    fetch(0);   // on their way while the scores are made
    if (live) {
#pragma unroll 8
      for (int d = 0; d < D; d += 4) {
        const float4 k4 = *reinterpret_cast<const float4 *>(kp + d);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float4 q4 = *reinterpret_cast<const float4 *>(&s_q[g][d]);
          sc[g] = fmaf(q4.x, k4.x, sc[g]);
          sc[g] = fmaf(q4.y, k4.y, sc[g]);
          sc[g] = fmaf(q4.z, k4.z, sc[g]);
          sc[g] = fmaf(q4.w, k4.w, sc[g]);
        }
      }
    }
    float pw[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float sv = live ? sc[g] * scale : kSeed;
      const float nm = fmaxf(mx[g], warp_max(sv));
      // fast exponentials (2^-21 relative): the scan is bound by instruction issue
      const float alpha = __expf(mx[g] - nm);
      pw[g] = live ? __expf(sv - nm) : 0.f;
      l[g] = fmaf(l[g], alpha, warp_sum(pw[g]));
      mx[g] = nm;
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        acc[g][e] *= alpha;
    }
    for (int t0 = 0; t0 < nk; t0 += VB) {
      if (t0 > 0)
        fetch(t0);
#pragma unroll
      for (int u = 0; u < VB; ++u)
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float pt = __shfl_sync(0xffffffffu, pw[g], t0 + u);
#pragma unroll
          for (int e = 0; e < VEC; ++e)
            acc[g][e] = fmaf(pt, vr[u][e], acc[g][e]);
        }
    }
  }
  __shared__ float s_m[WMAX][G], s_l[WMAX][G];
  __shared__ float s_acc[WMAX][G][D];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) {
      s_m[warp][g] = mx[g];
      s_l[warp][g] = l[g];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      s_acc[warp][g][lane * VEC + e] = acc[g][e];
  }
  __syncthreads();
  // [row][kv head][chunk][G][D] sums, then [..][G] pairs (max, sum of weights)
  const int64_t slot = ((int64_t)m * kv_heads + hk) * gridDim.z + sp;
  float *pout = part + slot * G * D;
  float2 *ml = reinterpret_cast<float2 *>(part + (int64_t)gridDim.x * kv_heads * gridDim.z * G * D);
  for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
    const int g = idx / D, d = idx - g * D;
    float M = kSeed;
    for (int w = 0; w < W; ++w)
      M = fmaxf(M, s_m[w][g]);
    float L = 0.f, A = 0.f;
    for (int w = 0; w < W; ++w) {
      const float b = expf(s_m[w][g] - M);   // a warp that saw no key: l = 0, acc = 0
      L = fmaf(s_l[w][g], b, L);
      A = fmaf(s_acc[w][g][d], b, A);
    }
    pout[idx] = A;
    if (d == 0)
      ml[slot * G + g] = make_float2(M, L);
  }
  // The CTA that finishes a row's last chunk folds the chunks in chunk order (the counter
  // returns to zero for the next launch).
  const int n = (len + chunk - 1) / chunk;     // chunks that hold keys of this row
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    int *cnt = counters + m * kv_heads + hk;
    const int prev = atomicAdd(cnt, 1);
    s_last = prev == n - 1;
    if (s_last)
      *cnt = 0;
  }
  __syncthreads();
  if (!s_last)
    return;
  __threadfence();
  // factors of the chunks first, then the sums, 8 chunks in flight
  const int64_t slot0 = slot - sp;
  float *factor = &s_acc[0][0][0];   // [n][G], n <= WMAX * D
  __shared__ float s_total[G];
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    float M = kSeed, L = 0.f;
#pragma unroll 8
    for (int c = 0; c < n; ++c)
      M = fmaxf(M, __ldcg(ml + (slot0 + c) * G + g).x);
#pragma unroll 8
    for (int c = 0; c < n; ++c) {
      const float2 v = __ldcg(ml + (slot0 + c) * G + g);
      const float b = expf(v.x - M);
      factor[c * G + g] = b;
      L = fmaf(v.y, b, L);
    }
    s_total[g] = L;
  }
  __syncthreads();
  const float4 *pin = reinterpret_cast<const float4 *>(part + slot0 * G * D);
  for (int idx = threadIdx.x; idx < G * D / 4; idx += blockDim.x) {
    const int g = idx / (D / 4);
    float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c0 = 0; c0 < n; c0 += 8) {
      float4 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        v[c] = c0 + c < n ? __ldcg(pin + (int64_t)(c0 + c) * (G * D / 4) + idx) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float b = c0 + c < n ? factor[(c0 + c) * G + g] : 0.f;
        A = make_float4(fmaf(v[c].x, b, A.x), fmaf(v[c].y, b, A.y), fmaf(v[c].z, b, A.z), fmaf(v[c].w, b, A.w));
      }
    }
    const float L = s_total[g];
    float *o = out + (int64_t)m * ldo + (int64_t)hk * G * D + 4 * idx;
    o[0] = __fdiv_rn(A.x, L);
    o[1] = __fdiv_rn(A.y, L);
    o[2] = __fdiv_rn(A.z, L);
    o[3] = __fdiv_rn(A.w, L);
  }
}

template <int G>
int launch_paged_split(const float *qkv, int64_t ld, const float *kp, const float *vp, float *out, int64_t ldo,
                       int kv_heads, int D, int page, const int32_t *row_seq, const int32_t *row_pos,
                       const int32_t *block_table, int table_stride, int M, float *part, int *counters, int chunks,
                       int chunk, cudaStream_t st) {
  dim3 grid(M, kv_heads, chunks);
  const int threads = min(256, chunk);   // a warp per 32 keys of the chunk (32 .. 256, a multiple of 32)
  if (D == 128)
    return launch_after(gqa_paged_split_kernel<G, 4>, grid, threads, 0, st, qkv, ld, kp, vp, part, kv_heads, page, row_seq, row_pos,
                        block_table, table_stride, chunk, counters, out, ldo);
  return launch_after(gqa_paged_split_kernel<G, 2>, grid, threads, 0, st, qkv, ld, kp, vp, part, kv_heads, page, row_seq, row_pos,
                        block_table, table_stride, chunk, counters, out, ldo);
}

// one first-maximum per row of a [rows, n] matrix (Sampler.h:101-104); 1024 threads per row,
// 16-byte loads when the rows allow it
__global__ void __launch_bounds__(1024) argmax_rows_kernel(const float *v, int64_t n, int32_t *out) {
  const float *row = v + (int64_t)blockIdx.x * n;
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  auto take = [&](float x, int i) {
    if (x > bv || (x == bv && i < bi)) {
      bv = x;
      bi = i;
    }
  };
  if ((n & 3) == 0 && ((uintptr_t)row & 15) == 0) {
    for (int64_t i = (int64_t)threadIdx.x * 4; i < n; i += (int64_t)blockDim.x * 4) {
      const float4 x = *reinterpret_cast<const float4 *>(row + i);
      take(x.x, (int)i);
      take(x.y, (int)i + 1);
      take(x.z, (int)i + 2);
      take(x.w, (int)i + 3);
    }
  } else {
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
      take(row[i], (int)i);
  }
  __shared__ float sv[32];
  __shared__ int si[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) {
      bv = ov;
      bi = oi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = bv;
    si[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (sv[w] > bv || (sv[w] == bv && si[w] < bi)) {
        bv = sv[w];
        bi = si[w];
      }
    out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
  }
}

} // namespace

int rope_kv_paged_launch(float *qkv, int64_t ld, float *k_pool, float *v_pool, const float *inv_freq,
                         const float *q_norm, const float *k_norm, float eps, int q_heads, int kv_heads, int D,
                         int page, const int32_t *row_seq, const int32_t *row_pos, const int32_t *block_table,
                         int table_stride, int M, cudaStream_t st) {
  return rope_rows_launch<true>(RopeRows{qkv, ld, k_pool, v_pool, inv_freq, q_norm, k_norm, eps, q_heads, kv_heads, D, 0, 0, page, row_seq, row_pos,
                               block_table, table_stride}, M, st);
}

int64_t gqa_paged_scratch_floats(int rows, int q_heads, int D, int max_context) {
  const int chunk = paged_chunk(max_context);
  const int chunks = (max_context + chunk - 1) / chunk;
  // one completion counter per (row, kv head) in front (zero between launches), then the partials
  return ((int64_t)rows * q_heads + 3) / 4 * 4 + (int64_t)rows * chunks * q_heads * (D + 2);
}

// scratch: gqa_paged_scratch_floats(scratch_rows, ..) floats whose first scratch_rows * q_heads
// words are zero, or null (then, and for more than scratch_rows or kPagedSplitRows rows, every
// row is scanned by one CTA)
int gqa_paged_launch(const float *qkv, int64_t ld, const float *k_pool, const float *v_pool, float *out, int64_t ldo,
                     int q_heads, int kv_heads, int D, int page, const int32_t *row_seq, const int32_t *row_pos,
                     const int32_t *block_table, int table_stride, int M, float *scratch, int scratch_rows,
                     int max_context, cudaStream_t st) {
  if (D != 64 && D != 128)
    return fail(B200_EINVAL, "gqa_paged: head_dim %d (64 or 128 supported)", D);
  constexpr int kPagedSplitRows = 256;
  const int chunk = paged_chunk(max_context);
  constexpr int kMostChunks = 512;   // whose factors fit the shared memory of the fold (131072 positions)
  const bool split = scratch != nullptr && M <= scratch_rows && M <= kPagedSplitRows && max_context > chunk &&
                     (max_context + chunk - 1) / chunk <= kMostChunks;
  int *counters = reinterpret_cast<int *>(scratch);
  float *part = scratch ? scratch + ((int64_t)scratch_rows * q_heads + 3) / 4 * 4 : nullptr;
  const int chunks = (max_context + chunk - 1) / chunk;
  switch (q_heads / kv_heads) {
#define B200_G(G_)                                                                                          \
  case G_:                                                                                                  \
    if (split)                                                                                              \
      return launch_paged_split<G_>(qkv, ld, k_pool, v_pool, out, ldo, kv_heads, D, page, row_seq, row_pos, \
                                    block_table, table_stride, M, part, counters, chunks, chunk, st);       \
    return launch_paged_attn<G_>(qkv, ld, k_pool, v_pool, out, ldo, kv_heads, D, page, row_seq, row_pos,    \
                                 block_table, table_stride, M, st);
    B200_G(1) B200_G(2) B200_G(3) B200_G(4) B200_G(6) B200_G(8)
#undef B200_G
  default:
    return fail(B200_EINVAL, "gqa_paged: group size %d not built", q_heads / kv_heads);
  }
}

int argmax_rows_launch(const float *v, int64_t n, int rows, int32_t *out, cudaStream_t st) {
  argmax_rows_kernel<<<rows, 1024, 0, st>>>(v, n, out);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

int embed_rows_launch(const float *table, const int32_t *tokens_dev, float *x, int64_t H, int M, cudaStream_t st) {
  if (H % 4 != 0)
    return fail(B200_EINVAL, "embed_rows: hidden size must be a multiple of 4");
  embed_rows_kernel<<<M, 128, 0, st>>>(table, tokens_dev, x, H);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

int rope_kv_rows_launch(float *qkv, int64_t ld, float *k_cache, float *v_cache, const float *inv_freq,
                        const float *q_norm, const float *k_norm, float eps, int q_heads, int kv_heads, int D,
                        int max_len, int pos0, int M, cudaStream_t st) {
  return rope_rows_launch<false>(RopeRows{qkv, ld, k_cache, v_cache, inv_freq, q_norm, k_norm, eps, q_heads, kv_heads, D, max_len, pos0, 0, nullptr,
                               nullptr, nullptr, 0}, M, st);
}

int gqa_prefill_launch(const float *qkv, int64_t ld, const float *kc, const float *vc, float *out, int64_t ldo,
                       int q_heads, int kv_heads, int D, int max_len, int pos0, int M, cudaStream_t st) {
  if (D != 64 && D != 128)
    return fail(B200_EINVAL, "gqa_prefill: head_dim %d (64 or 128 supported)", D);
  switch (q_heads / kv_heads) {
#define B200_G(G_)                                                                                      \
  case G_:                                                                                              \
    return launch_prefill_attn<G_>(qkv, ld, kc, vc, out, ldo, q_heads, kv_heads, D, max_len, pos0, M, st);
    B200_G(1) B200_G(2) B200_G(3) B200_G(4) B200_G(6) B200_G(8)
#undef B200_G
  default:
    return fail(B200_EINVAL, "gqa_prefill: group size %d not built", q_heads / kv_heads);
  }
}

} // namespace b200
