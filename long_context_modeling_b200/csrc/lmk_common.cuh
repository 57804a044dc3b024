// What the landmark scan, its tensor-core form and the merges share: candidate keys, sorted lists, the outputs of a row.
#pragma once

#include "gca_common.cuh"

namespace gca {

constexpr int MAXK = 32;

__device__ __forceinline__ unsigned orderable(float s) {
  const unsigned u = __float_as_uint(s);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_orderable(unsigned o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ unsigned long long make_key(float score, unsigned gidx) {
  return ((unsigned long long)orderable(score) << 32) | (unsigned long long)(0xffffffffu - gidx);
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Insert `key` into the descending list held one element per lane.  Warp-uniform call.
__device__ __forceinline__ void list_insert(unsigned long long& mine, unsigned long long key, int lane) {
  const bool lower = mine < key;
  const unsigned long long up = __shfl_up_sync(0xffffffffu, mine, 1);
  const int lower_prev = __shfl_up_sync(0xffffffffu, (int)lower, 1);
  if (lower) mine = (lane > 0 && lower_prev) ? up : key;
}

__device__ __forceinline__ void unpack8(const uint4& v, float f[8]) {
  f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
  f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
  f[4] = __uint_as_float(v.z << 16); f[5] = __uint_as_float(v.z & 0xffff0000u);
  f[6] = __uint_as_float(v.w << 16); f[7] = __uint_as_float(v.w & 0xffff0000u);
}

struct FinalParams {
  const unsigned long long* keys;   // (R, P)
  unsigned long long* out_keys;
  int32_t* out_indices;
  float* out_scores;
  float* out_weights;
  int32_t* out_nvalid;
  int32_t* kept_indices = nullptr;  // a second copy of indices and weights, or nullptr
  float* kept_weights = nullptr;
  // optional recompute of noise-free scores (per-sequence mode with noise)
  const __nv_bfloat16* lq;
  const __nv_bfloat16* lk;
  long long qbs, qrs, kbs, krs, e_base;
  int Cq, D, score_round;
  float scale;
  int R, P, K;
  int lists;                        // keys come as P / K descending lists of K (the scan's own output)
};

// The scan's dot product: lane l sums the pieces l, l + 32, ... of 8 elements in order, then the butterfly.  Every lane gets it.
__device__ __forceinline__ float exact_dot(const __nv_bfloat16* a, const __nv_bfloat16* b, int pieces, int lane) {
  float acc = 0.f;
  for (int c = lane; c < pieces; c += 32) {
    float af[8], bf[8];
    unpack8(*reinterpret_cast<const uint4*>(a + c * 8), af);
    unpack8(*reinterpret_cast<const uint4*>(b + c * 8), bf);
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) acc = fmaf(af[jj], bf[jj], acc);
  }
#pragma unroll
  for (int of = 16; of > 0; of >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, of);
  return acc;
}

// One warp writes the outputs of a row: lane i holds the i-th best key (0 = none) and its noise-free score.
__device__ __forceinline__ void emit_scored(const FinalParams& p, long long row, unsigned long long m, float score, int lane) {
  const bool valid = lane < p.K && m != 0ull;
  const int idx = valid ? (int)(0xffffffffu - (unsigned)(m & 0xffffffffull)) : -1;
  if (!valid) score = -INFINITY;
  // softmax over the valid slots
  float mx = valid ? score : -INFINITY;
#pragma unroll
  for (int of = 16; of > 0; of >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, of));
  float ex = valid ? expf(score - mx) : 0.f;
  float sum = ex;
#pragma unroll
  for (int of = 16; of > 0; of >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, of);
  const float wgt = (valid && sum > 0.f) ? ex / sum : 0.f;
  const unsigned nv = __popc(__ballot_sync(0xffffffffu, valid));
  if (lane < p.K) {
    const long long o = row * p.K + lane;
    if (p.out_keys) p.out_keys[o] = m;
    if (p.out_indices) p.out_indices[o] = idx;
    if (p.out_scores) p.out_scores[o] = score;
    if (p.out_weights) p.out_weights[o] = wgt;
    if (p.kept_indices) { p.kept_indices[o] = idx; p.kept_weights[o] = wgt; }
  }
  if (lane == 0 && p.out_nvalid) p.out_nvalid[row] = (int)nv;
}

// The same from the keys alone; when the selection used noisy scores (p.lq given) the noise-free score of every winner is
// computed again in the scan's order.
__device__ __forceinline__ void emit_row(const FinalParams& p, long long row, unsigned long long m, int lane) {
  const bool valid = lane < p.K && m != 0ull;
  const int idx = valid ? (int)(0xffffffffu - (unsigned)(m & 0xffffffffull)) : -1;
  float score = valid ? from_orderable((unsigned)(m >> 32)) : -INFINITY;
  if (p.lq) {
    const long long n = row / p.Cq, r = row % p.Cq;
#pragma unroll 4
    for (int i = 0; i < p.K; ++i) {                         // no branch on the slot: the loads of four winners overlap
      const int won = __shfl_sync(0xffffffffu, idx, i);
      const long long wi = won < 0 ? p.e_base : won;
      const float acc = exact_dot(p.lq + n * p.qbs + r * p.qrs, p.lk + n * p.kbs + (wi - p.e_base) * p.krs, p.D >> 3, lane);
      const float s = p.score_round ? round_bf16(round_bf16(acc) * p.scale) : acc * p.scale;
      if (lane == i && won >= 0) score = s;
    }
  }
  emit_scored(p, row, m, score, lane);
}

}  // namespace gca
