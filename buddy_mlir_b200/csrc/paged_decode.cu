// Attention of one decode step of many sequences over the page pool, with what comes before it: head norm and RoPE of q and k, and
// the new K and V rows' way to their pages (subgraph0_decode_simplify.mlir:52-59, 86-142; the recurrence of
// frontend/Python/ops/tosa.py:14245-14594).  Every row of the batch is the newest position of a sequence of its own.
//
// What bounds it is a chain of latencies, not the 19 MB of a layer (24 sequences of 32..700 positions, 12 heads on 2, D = 128: 3 us
// of HBM).  So the keys of a row are dealt evenly to the 8 warps of up to 8 CTAs of a cluster, four keys at a time: a lane owns
// D / 32 dims, K and V rows are whole 512-byte loads, and 24 scores (4 keys x 6 heads) are summed across the lanes together with 27
// shuffles.  The first rows are requested before the kernel waits for the one before it: nothing of this pass writes them.  (Sending the
// others to L2 there gains nothing for 24 rows of 500 keys, and costs 16 rows of 8000 17 us a layer.)  Warps
// meet in shared memory, CTAs in that of the cluster, each completing its share of the output.
// That step of 24 sequences, a layer, from q|k|v on: 32 us for RoPE, a scan of 32 keys per warp with a lane per key and a fold
// through L2; 14 us here, of which 8 for the longest rows' five turns of a warp (about 450 instructions each), 3 for the sums.
// (Chunks of 96 keys of all rows, and the CTA that finishes a row's last one adding them up: 18 us, six of them for that; CTAs of four
// warps, eight to a row: as long; a bulk prefetch per row holds its warp a lane at a time.)
// Scores are scaled in q, in powers of two, and all exponentials are ex2.approx (2 ulp), those of the sums' factors too.  Relative error
// against f64 (2-norm, Gaussian inputs; in brackets q six times as large) here / in the kernels that it stands in for: 24 rows of 1..700 keys,
// 12 heads on 2, 1.5e-7 / 3.3e-7 (3.2e-7 / 1.2e-6); 300 rows, where each had one CTA and expf, 1.5e-7 / 1.6e-7 (3.3e-7 / 4.1e-7);
// contexts of up to 30 keys 9.5e-8 / 9.2e-8; 300 rows of up to 97, 8 heads of 64, 1.02e-7 / 1.01e-7 (2.43e-7 / 2.31e-7).  (With expf of scores scaled after the sum 1.4e-7, 1.4e-7, 9.3e-8, but 3.7e-7 for the large
// ones, and 3 % longer, up to 17; exp2f gives the bits of ex2.)
#include "common.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr float kSeed = -1.0e30f;
constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kKeys = 4;             // of a warp at a time
constexpr int kMaxCluster = 8;
constexpr int kMaxRange = 1024;      // keys of a CTA
constexpr int kCtas = 148;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float from_cta(const float *p, int rank) {   // shared memory of the cluster's CTA `rank`
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 from_cta4(const float *p, int rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 fma4(float4 a, float b, float4 c) {
  return make_float4(fmaf(a.x, b, c.x), fmaf(a.y, b, c.y), fmaf(a.z, b, c.z), fmaf(a.w, b, c.w));
}
__device__ __forceinline__ void store_over(float *p, float4 a, float l) {   // (rows of the output need not be aligned)
  p[0] = __fdiv_rn(a.x, l);
  p[1] = __fdiv_rn(a.y, l);
  p[2] = __fdiv_rn(a.z, l);
  p[3] = __fdiv_rn(a.w, l);
}
__device__ __forceinline__ void sync_cluster() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int VEC> struct Vec {
  float v[VEC];
  __device__ __forceinline__ void load(const float *p) {
    if constexpr (VEC == 4) {
      const float4 a = *reinterpret_cast<const float4 *>(p);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
      const float2 a = *reinterpret_cast<const float2 *>(p);
      v[0] = a.x; v[1] = a.y;
    }
  }
  __device__ __forceinline__ void store(float *p) const {
    if constexpr (VEC == 4)
      *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else
      *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
  }
};

// N values summed across the lanes: while N is even a step halves them (a lane's bit says which half it keeps), so that the
// lane is left with N >> halvings(N) sums, those of values i + (N >> 1) * bit 4 + (N >> 2) * bit 3 + ..
__host__ __device__ constexpr int halvings(int n) {
  int h = 0;
  while (h < 5 && n % 2 == 0) {
    n /= 2;
    ++h;
  }
  return h;
}
template <int N, int BIT = 16> __device__ __forceinline__ void sum_lanes(float *v) {
  if constexpr (BIT > 0) {
    if constexpr (N % 2 == 0) {
      const bool up = threadIdx.x & BIT;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        const float give = up ? v[i] : v[i + N / 2], keep = up ? v[i + N / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, BIT);
      }
      sum_lanes<N / 2, BIT / 2>(v);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i)
        v[i] += __shfl_xor_sync(0xffffffffu, v[i], BIT);
      sum_lanes<N, BIT / 2>(v);
    }
  }
}

struct PagedParams {
  const float *qkv;            // [M][ld]: q heads, k heads, v heads
  int64_t ld;
  float *k_pool, *v_pool;      // [pages][kv_heads][page][D]
  const float *inv_freq, *q_norm, *k_norm;
  float eps;
  int kv_heads, page;
  const int32_t *row_seq, *row_pos, *block_table;
  int table_stride;
  float *out;                  // [M][ldo]
  int64_t ldo;
};

// grid (cluster, kv heads, rows), clusters along x
template <int G, int VEC>
__global__ void __launch_bounds__(kThreads, 2) paged_decode_kernel(const __grid_constant__ PagedParams p) {
  constexpr int D = 32 * VEC, N = kKeys * G, H = halvings(N), LEFT = N >> H;   // scores, and those a lane is left with
  __shared__ int s_row[kMaxRange];
  __shared__ __align__(16) float s_new[3][D], s_acc[kWarps][G][D], s_sum[G][D];
  __shared__ float s_m[kWarps][G], s_l[kWarps][G], s_max[G], s_total[G];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m = blockIdx.z, hk = blockIdx.y, C = gridDim.x, sp = blockIdx.x;
  kernel_go();
  const int pos = p.row_pos[m], len = pos + 1, per = ((len + C - 1) / C + kKeys - 1) / kKeys * kKeys;
  const int j0 = min(sp * per, len), j1 = min(len, j0 + per);   // (only the range with the newest key may end within a warp's four)
  const int32_t *table = p.block_table + (int64_t)p.row_seq[m] * p.table_stride;
  for (int j = j0 + threadIdx.x; j < j1; j += kThreads)
    s_row[j - j0] = (table[j / p.page] * p.kv_heads + hk) * p.page + j % p.page;
  float cs[VEC], sn[VEC];   // of this lane's dims: pairs (j, j + D / 2) are 16 lanes apart
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    const float th = __fmul_rn(__ldg(p.inv_freq + ((lane * VEC + e) & (D / 2 - 1))), (float)pos);
    cs[e] = cosf(th);
    sn[e] = lane < 16 ? -sinf(th) : sinf(th);
  }
  __syncthreads();
  Vec<VEC> k[kKeys], v[kKeys];
  auto request = [&](int jb) {   // (the newest row is not there yet, or is what it was: its values come from shared memory)
#pragma unroll
    for (int u = 0; u < kKeys; ++u) {
      const int64_t at = (int64_t)s_row[min(jb + u, j1 - 1) - j0] * D + lane * VEC;
      k[u].load(p.k_pool + at);
      v[u].load(p.v_pool + at);
    }
  };
  int jb = j0 + warp * kKeys;
  if (jb < j1)
    request(jb);
  kernel_wait();

  // ---- q heads; the CTA with the newest position: k and v (first warp) --------------------------------------------------------
  auto rotate = [&](Vec<VEC> &x, const float *norm) {
    if (norm != nullptr) {
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        ss = fmaf(x.v[e], x.v[e], ss);
      const float r = rsqrtf(__fadd_rn(__fmul_rn(warp_sum(ss), 1.0f / (float)D), p.eps));
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        x.v[e] = __fmul_rn(__ldg(norm + lane * VEC + e), __fmul_rn(x.v[e], r));
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const float other = __shfl_xor_sync(0xffffffffu, x.v[e], 16);
      x.v[e] = __fadd_rn(__fmul_rn(x.v[e], cs[e]), __fmul_rn(other, sn[e]));
    }
  };
  const float *row = p.qkv + (int64_t)m * p.ld + lane * VEC;
  const int q_dims = p.kv_heads * G * D;
  Vec<VEC> q[G], nk, nv;
#pragma unroll
  for (int g = 0; g < G; ++g)
    q[g].load(row + (hk * G + g) * D);
  if (j1 == len && j0 < len && warp == 0) {
    nk.load(row + q_dims + hk * D);
    nv.load(row + q_dims + (p.kv_heads + hk) * D);
    rotate(nk, p.k_norm);
    const int64_t at = (int64_t)s_row[pos - j0] * D + lane * VEC;
    nk.store(p.k_pool + at);
    nv.store(p.v_pool + at);
    nk.store(&s_new[0][lane * VEC]);
    nv.store(&s_new[1][lane * VEC]);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      s_new[2][lane * VEC + e] = 0.f;
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    rotate(q[g], p.q_norm);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      q[g].v[e] *= rsqrtf((float)D) * 1.4426950408889634f;   // scores in powers of two
  }
  __syncthreads();

  // ---- this warp's keys --------------------------------------------------------------------------------------------------------
  // After sum_lanes a lane has the scores of key lane / 8 and LEFT heads from `head` on; heads of lanes that differ only in the
  // bits below are the same.
  int head = 0;
#pragma unroll
  for (int b = 2; b < H; ++b)
    head += (lane >> (4 - b) & 1) * (N >> (b + 1));
  float acc[G][VEC] = {}, mx[LEFT], l[LEFT];
#pragma unroll
  for (int i = 0; i < LEFT; ++i) {
    mx[i] = kSeed;
    l[i] = 0.f;
  }
  auto lane_of = [](int u, int g) {   // a lane that has the score of key u and head g (in register g % LEFT)
    int at = u << 3, first = 0;
    for (int b = 2; b < H; ++b)
      if (g >= first + (N >> (b + 1))) {
        first += N >> (b + 1);
        at |= 16 >> b;
      }
    return at;
  };
#pragma unroll 1
  for (; jb < j1; jb += kWarps * kKeys) {
    // the newest key (its row in the pool may be anything yet), and in the place of keys beyond it, whose weight is zero, a value of zero
    if (j1 == len && jb + kKeys > pos) {
#pragma unroll
      for (int u = 0; u < kKeys; ++u)
        if (jb + u >= pos) {
          k[u].load(&s_new[0][lane * VEC]);
          v[u].load(&s_new[jb + u > pos ? 2 : 1][lane * VEC]);
        }
    }
    float sc[N];
#pragma unroll
    for (int u = 0; u < kKeys; ++u)
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          a = fmaf(q[g].v[e], k[u].v[e], a);
        sc[u * G + g] = a;
      }
    Vec<VEC> cv[kKeys];
#pragma unroll
    for (int u = 0; u < kKeys; ++u)
      cv[u] = v[u];
    if (jb + kWarps * kKeys < j1)
      request(jb + kWarps * kKeys);
    sum_lanes<N>(sc);
    const bool live = jb + (lane >> 3) < j1;
    float alpha[LEFT], pw[LEFT];
    bool grows = false;
#pragma unroll
    for (int i = 0; i < LEFT; ++i) {
      const float s = live ? sc[i] : kSeed;
      float nm = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, 16));
      nm = fmaxf(mx[i], fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, 8)));
      grows = grows || nm > mx[i];
      alpha[i] = ex2(mx[i] - nm);
      pw[i] = live ? ex2(s - nm) : 0.f;
      l[i] = fmaf(l[i], alpha[i], pw[i]);
      mx[i] = nm;
    }
    if (__any_sync(0xffffffffu, grows)) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float a = __shfl_sync(0xffffffffu, alpha[g % LEFT], lane_of(0, g));
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          acc[g][e] *= a;
      }
    }
#pragma unroll
    for (int u = 0; u < kKeys; ++u)
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float w = __shfl_sync(0xffffffffu, pw[g % LEFT], lane_of(u, g));
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          acc[g][e] = fmaf(w, cv[u].v[e], acc[g][e]);
      }
  }

  // ---- the warps' sums, then the CTAs' -------------------------------------------------------------------------------------------
#pragma unroll
  for (int i = 0; i < LEFT; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 16);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 8);
    if (lane < 8) {   // (lanes with the same heads write the same)
      s_m[warp][head + i] = mx[i];
      s_l[warp][head + i] = l[i];
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    Vec<VEC> a;
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      a.v[e] = acc[g][e];
    a.store(&s_acc[warp][g][lane * VEC]);
  }
  __syncthreads();
  float *out = p.out + (int64_t)m * p.ldo + (int64_t)hk * G * D;
#pragma unroll 1
  for (int i = threadIdx.x; i < G * D / 4; i += kThreads) {
    const int g = i / (D / 4), d = i % (D / 4) * 4;
    float M = kSeed, L = 0.f;
    float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWarps; ++w)
      M = fmaxf(M, s_m[w][g]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {   // (a warp that saw no key: sums of zero)
      const float b = ex2(s_m[w][g] - M);
      L = fmaf(s_l[w][g], b, L);
      A = fma4(*reinterpret_cast<const float4 *>(&s_acc[w][g][d]), b, A);
    }
    if (C == 1) {
      store_over(out + 4 * i, A, L);
    } else {
      *reinterpret_cast<float4 *>(&s_sum[g][d]) = A;
      if (d == 0) {
        s_max[g] = M;
        s_total[g] = L;
      }
    }
  }
  if (C == 1)
    return;
  sync_cluster();
  for (int i = G * D / 4 * sp / C + threadIdx.x; i < G * D / 4 * (sp + 1) / C; i += kThreads) {
    const int g = i / (D / 4);
    float cm[kMaxCluster], cl[kMaxCluster], M = kSeed, L = 0.f;
    float4 ca[kMaxCluster], A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int z = 0; z < kMaxCluster; ++z) {
      cm[z] = z < C ? from_cta(&s_max[g], z) : kSeed;
      cl[z] = z < C ? from_cta(&s_total[g], z) : 0.f;
      ca[z] = z < C ? from_cta4(&s_sum[0][0] + 4 * i, z) : make_float4(0.f, 0.f, 0.f, 0.f);
      M = fmaxf(M, cm[z]);
    }
#pragma unroll
    for (int z = 0; z < kMaxCluster; ++z) {
      const float b = ex2(cm[z] - M);
      L = fmaf(cl[z], b, L);
      A = fma4(ca[z], b, A);
    }
    store_over(out + 4 * i, A, L);
  }
  sync_cluster();   // none ends while another reads its sums
}

// CTAs per (row, kv head): enough for every SM, all of them at once, and at least 32 keys each in the longest row.
int cluster_size(int M, int kv_heads, int longest) {
  int c = 1;
  while (c < kMaxCluster && (int64_t)M * kv_heads * c < kCtas && longest > 32 * c)
    c *= 2;
  return c;
}

// A CTA's range of keys is a chain of turns of 32 (0.5 to 1.2 us each, 2 at eight heads of 128, whose registers do not all fit), and no
// more than 8 CTAs share a row: with few rows of long contexts the general kernels, which cut them in chunks of 256 keys over the whole
// chip, are done sooner.  us a layer here / there, RoPE included, caches from memory; q heads on kv heads of 128:
//   12 on 2   2 rows of 4000 21 / 26, of 8000 38 / 30; 4 of 8000 41 / 33; 8 of 4000 31 / 31, of 8000 54 / 58; 16 of 8000 56 / 110
//   32 on 8   2 rows of 4000 22 / 28, of 8000 38 / 53      4 on 2   2 of 4000 16 / 21, of 8000 29 / 25; 8 of 8000 34 / 47
//   8 on 1    2 rows of 2000 19 / 24, of 4000 34 / 24; 16 of 2000 28 / 29, of 3000 39 / 34; 24 of 3000 40 / 35, of 4000 51 / 60;
//             37 of 1000 28 / 32, of 2000 50 / 33; 64 of 4000 93 / 116; 100 of 1000 51 / 61, of 2000 93 / 88
bool ranges_pay(int G, int D, int ctas, int range, int longest) {
  if (G == 8 && D == 128)
    return range <= 320 || longest <= 1024 || ctas >= 256;
  return range <= 512 || ctas >= 128;
}

} // namespace

bool paged_decode_takes(const float *qkv, int64_t ld, const float *k_pool, const float *v_pool, int q_heads, int kv_heads, int D, int M,
                        int longest) {
  const int G = q_heads / kv_heads, C = cluster_size(M, kv_heads, longest);
  return (D == 64 || D == 128) && q_heads == G * kv_heads && (G == 1 || G == 2 || G == 3 || G == 4 || G == 6 || G == 8) && M <= 65535 &&
         kv_heads <= 65535 && (longest + C - 1) / C <= kMaxRange && ranges_pay(G, D, M * kv_heads * C, (longest + C - 1) / C, longest) && (ld & 3) == 0 &&
         (((uintptr_t)qkv | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0;
}

int paged_decode_launch(const float *qkv, int64_t ld, float *k_pool, float *v_pool, float *out, int64_t ldo, const float *inv_freq,
                        const float *q_norm, const float *k_norm, float eps, int q_heads, int kv_heads, int D, int page,
                        const int32_t *row_seq, const int32_t *row_pos, const int32_t *block_table, int table_stride, int M, int longest,
                        cudaStream_t st) {
  const PagedParams p{qkv, ld, k_pool, v_pool, inv_freq, q_norm, k_norm, eps, kv_heads, page, row_seq, row_pos, block_table, table_stride, out, ldo};
  const int C = cluster_size(M, kv_heads, longest);
  const dim3 grid(C, kv_heads, M);
  switch (q_heads / kv_heads) {
#define B200_G(G_)                                                                                                   \
  case G_:                                                                                                           \
    return D == 128 ? launch_after_clusters(C, paged_decode_kernel<G_, 4>, grid, kThreads, 0, st, p)                 \
                    : launch_after_clusters(C, paged_decode_kernel<G_, 2>, grid, kThreads, 0, st, p);
    B200_G(1) B200_G(2) B200_G(3) B200_G(4) B200_G(6) B200_G(8)
#undef B200_G
  default:
    return fail(B200_EINVAL, "paged decode: group size %d not built", q_heads / kv_heads);
  }
}

} // namespace b200
