// Parameters of the persistent decode-step kernel (decode.cu).
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int kDecWarps = 16;
constexpr int kDecThreads = kDecWarps * 32;
constexpr int kDecMaxK = 12288;        // longest activation vector a CTA stages 
constexpr int kDecMaxSplits = 32;      // key ranges per kv head (one lane each when they are folded)
constexpr int kDecTraceSlots = 64;     // trace points per (CTA, layer)
constexpr int kDecBlockBytes = 2048;   // weights of one stream block
// Stream blocks in flight per warp (int4 models: the activation vectors of the large model leave room for three).
__host__ __device__ constexpr int dec_slots(int mode) { return mode == 2 ? 3 : 4; }
constexpr int kDecScaleBytes = 64;     // int4: behind them, 16 rows x 2 groups of f16 scales

// One projection as the kernel sees it: tiles of 16 rows, dealt out to the CTAs in contiguous ranges; a tile is
// `blocks` stream blocks long (int8: 128 k each, int4: 256 k, f32: 32 k; K is padded with zero weights).
struct DecPhase {
  int kind, K, N, tiles, blocks;
};
// What differs between layers.
struct DecLayer {
  const float *in_norm, *post_norm, *q_norm, *k_norm;
  const float *scale[4];   // int8: [N] per projection (q|k|v, o, gate|up, down)
  const float *qkv_bias;
  float *k_cache, *v_cache;
};

struct DecParams {
  const uint8_t *stream;        // every warp's private weight stream, back to back
  const int64_t *warp_off;      // [grid * 16] start of each warp's stream
  DecPhase phase[5];            // q|k|v, o, gate|up (interleaved pairs), down, lm_head
  const DecLayer *layers;
  const float *lm_scale, *final_norm, *embed, *inv_freq;
  int H, F, V, qh, kvh, L, max_len;
  int block_bytes;
  int union_bytes, part_rows;   // shared memory: activation planes / attention scratch; partial sums
  float eps;
  // tagged (value, tag) activation buffers, two copies each (layer parity)
  uint2 *ll_qkv;                // [2][QD + 2*KD]
  uint2 *ll_attn;               // [2][QD]
  uint2 *ll_xb;                 // [2][H]   residual stream after attention
  uint2 *ll_mid;                // [2][F]   silu(gate) * up
  uint2 *ll_xa;                 // [2][H]   residual stream after the MLP
  uint2 *ll_part;               // [2][qh][kDecMaxSplits][130] attention split partials: acc, m, l
  uint2 *ll_cand;               // [grid][2] per-CTA argmax candidates (value, index)
  float *logits;
  float *kv_stage;              // [2*L][kvh*D] rows written this step
  // the same in page-locked host memory, or null.  Written beside the step's own work: 608 KB of logits cross the bus while the
  // lm_head streams, where a copy behind the kernel took 15 us (and one of the rows 3)
  float *logits_host, *rows_host;
  int32_t *state;               // token, pos, next, count, launches completed
  int32_t *history;
  int history_cap;
  int *error;                   // 0, or the code of the first wait that gave up
  long long *trace;             // optional [grid/stride][L+1][kDecTraceSlots] SM-clock timeline, or null
  int trace_stride;
};

int dec_block_k(int kind);                           // k per stream block
size_t dec_union_bytes(const DecPhase *ph, int G);   // shared memory of the planes / attention scratch
size_t dec_shared_bytes(const DecParams &p);
bool dec_group_built(int G);                         // q heads per kv head the kernel is compiled for
// The blocks of every CTA's every warp of one projection, from the packed rows (all layers' streams share one layout;
// `skip` = bytes of the stream before this projection, per warp: [grid * 16]).
int dec_build_phase(const b200_weight *w, const DecPhase &ph, int grid, int block_bytes, const int64_t *warp_off,
                    const int64_t *skip, uint8_t *stream, cudaStream_t st);
int dec_launch(const DecParams &p, int grid, size_t smem, cudaStream_t st);

// Contiguous share of n things for part i of parts.
__host__ __device__ inline int share_begin(int n, int i, int parts) { return (int)((int64_t)n * i / parts); }

// A CTA's nb blocks of a projection, cut into contiguous shares of its warps (of nb warps when there are fewer blocks):
// first block of warp w, and the warp that owns block b.
__host__ __device__ inline int warp_begin(int nb, int w) {
  const int n = nb < kDecWarps ? nb : kDecWarps;
  return w < n ? share_begin(nb, w, n) : nb;
}
__host__ __device__ inline int warp_of(int nb, int b) {
  const int n = nb < kDecWarps ? nb : kDecWarps;
  return (n * b + n - 1) / nb;
}

} // namespace b200
