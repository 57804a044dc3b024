// Gradient of the retrieval weights into the landmarks (model/DRT.py:626: softmax over the gathered scores; the
// reference gets it from autograd through einsum, gather and the index_put of the gathered rows).
//
//   w[c, :] = softmax_k(q_c . m_idx(c,k) / sqrt(D))   ->   ds[c, k] = w (dw - sum_k w dw) / sqrt(D)
//   dq[c]   = sum_k ds[c, k] m_idx(c,k)                    dm[e] = sum over (c, k) with idx(c, k) = e of ds[c, k] q_c
//
// One launch, a warp per row of dq and a block per row of dm, no atomics, sums in a fixed order.  The rows of dm find their retrievers by
// reading the index array themselves (K ints per query row, from the first row that can see the landmark on): building
// an inverse index first costs more launches than that read as long as a sequence has a few thousand chunks.
// What bounds it is latency, one L2 round trip per retriever, so the four warps of a row's block share its retrievers (an
// early landmark has many times the average), collect them first and take them four at a time.  At 8 x 260 chunks, K = 8: torch's gather + einsum + softmax and their backward 45 launches, ~330 us.
#include "gca_common.cuh"

namespace gca {

namespace {

constexpr int GRAD_WARPS = 4, BATCH = 4, SCAN = 4, LIST = SCAN * 32 + BATCH;

struct GradParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* m;
  const int32_t* indices;      // (N, Cq, K), -1 = padding
  const float* weights;        // (N, Cq, K)
  const float* dw_rows;        // (N, rows_a, K) by strides, or nullptr: the gradient of the first rows_a rows
  const float* dw_all;         // (N, Cq, K) by strides, or nullptr
  __nv_bfloat16* dq;
  __nv_bfloat16* dm;
  long long qbs, qrs, mbs, mrs, a_s[3], b_s[3];
  long long q_pos0;
  int N, Cq, E, D, K, rows_a;
  float scale;
};

__device__ __forceinline__ void fma8(float* acc, float s, const uint4& v) {
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc[2 * i] = fmaf(s, __uint_as_float(w[i] << 16), acc[2 * i]);
    acc[2 * i + 1] = fmaf(s, __uint_as_float(w[i] & 0xffff0000u), acc[2 * i + 1]);
  }
}

// lane k < K: ds of slot k of query row (n, c)
__device__ __forceinline__ float slot_grads(const GradParams& p, int n, int c, int lane) {
  float w = 0.f, d = 0.f;
  if (lane < p.K) {
    w = p.weights[((long long)n * p.Cq + c) * p.K + lane];
    if (p.dw_rows && c < p.rows_a) d = p.dw_rows[n * p.a_s[0] + c * p.a_s[1] + lane * p.a_s[2]];
    if (p.dw_all) d += p.dw_all[n * p.b_s[0] + c * p.b_s[1] + lane * p.b_s[2]];
  }
  float t = w * d;
#pragma unroll
  for (int of = 16; of > 0; of >>= 1) t += __shfl_xor_sync(0xffffffffu, t, of);
  return w * (d - t) * p.scale;
}

template <int NP>
__device__ __forceinline__ void store_row(__nv_bfloat16* dst, const float (*acc)[8], int pieces, int lane) {
#pragma unroll
  for (int pp = 0; pp < NP; ++pp) {
    const int c = lane + 32 * pp;
    if (c >= pieces) continue;
    unsigned o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(acc[pp][2 * i], acc[pp][2 * i + 1]);
      o[i] = *reinterpret_cast<const unsigned*>(&b);
    }
    *reinterpret_cast<uint4*>(dst + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int NP>
__global__ void __launch_bounds__(GRAD_WARPS * 32)
lmk_grad_kernel(GradParams p) {
  __shared__ int list_all[GRAD_WARPS][LIST];
  __shared__ __align__(16) float sums[GRAD_WARPS - 1][NP * 256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pieces = p.D >> 3;
  int* list = list_all[warp];
  // the rows of dm first: the longer units
  const long long m_blocks = p.dm ? (long long)p.N * p.E : 0;
  float acc[NP][8];
#pragma unroll
  for (int pp = 0; pp < NP; ++pp)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[pp][i] = 0.f;
  if (blockIdx.x >= m_blocks) {
    const long long u = (blockIdx.x - m_blocks) * GRAD_WARPS + warp;
    if (u >= (long long)p.N * p.Cq) return;
    const int n = (int)(u / p.Cq), c = (int)(u % p.Cq);
    const float ds = slot_grads(p, n, c, lane);
    const int id = lane < p.K ? p.indices[((long long)n * p.Cq + c) * p.K + lane] : -1;
#pragma unroll 4
    for (int k = 0; k < p.K; ++k) {
      const int e = __shfl_sync(0xffffffffu, id, k);
      const float s = __shfl_sync(0xffffffffu, ds, k);
      if (e < 0 || e >= p.E) continue;
#pragma unroll
      for (int pp = 0; pp < NP; ++pp)
        if (lane + 32 * pp < pieces) fma8(acc[pp], s, *reinterpret_cast<const uint4*>(p.m + n * p.mbs + e * p.mrs + (lane + 32 * pp) * 8));
    }
    store_row<NP>(p.dq + ((long long)n * p.Cq + c) * p.D, acc, pieces, lane);
    return;
  }
  const int e = (int)(blockIdx.x / p.N), n = (int)(blockIdx.x % p.N);
  const long long first = e - p.q_pos0 + 1;               // row c sees landmark e iff e < q_pos0 + c
  const int32_t* ids = p.indices + (long long)n * p.Cq * p.K;
  const int total = p.Cq * p.K;
  int have = 0;
  auto drain = [&](int upto) {                              // list[0 .. upto) in order, BATCH rows in flight
    for (int b = 0; b < upto; b += BATCH) {
      uint4 row[BATCH][NP];
      float s[BATCH];
#pragma unroll
      for (int x = 0; x < BATCH; ++x) {
        const int slot = b + x < upto ? list[b + x] : -1;
        s[x] = 0.f;
        if (slot < 0) continue;                             // warp-uniform
        const int c = slot / p.K;
#pragma unroll
        for (int pp = 0; pp < NP; ++pp) {
          row[x][pp] = make_uint4(0, 0, 0, 0);
          if (lane + 32 * pp < pieces) row[x][pp] = *reinterpret_cast<const uint4*>(p.q + n * p.qbs + c * p.qrs + (lane + 32 * pp) * 8);
        }
        s[x] = __shfl_sync(0xffffffffu, slot_grads(p, n, c, lane), slot - c * p.K);
      }
#pragma unroll
      for (int x = 0; x < BATCH; ++x)
        if (b + x < upto) {
#pragma unroll
          for (int pp = 0; pp < NP; ++pp) fma8(acc[pp], s[x], row[x][pp]);
        }
    }
  };
  for (int i0 = (int)(first > 0 ? first : 0) * p.K + warp * SCAN * 32; i0 < total; i0 += GRAD_WARPS * SCAN * 32) {
    int id[SCAN];
#pragma unroll
    for (int x = 0; x < SCAN; ++x) id[x] = i0 + x * 32 + lane < total ? ids[i0 + x * 32 + lane] : -1;
#pragma unroll
    for (int x = 0; x < SCAN; ++x) {
      const unsigned b = __ballot_sync(0xffffffffu, id[x] == e);
      if (id[x] == e) list[have + __popc(b & ((1u << lane) - 1u))] = i0 + x * 32 + lane;
      have += __popc(b);
    }
    __syncwarp();
    if (have >= BATCH) {                                    // whole batches; the remainder moves to the front
      const int whole = have / BATCH * BATCH;
      drain(whole);
      __syncwarp();
      const int rest = have - whole, moved = lane < rest ? list[whole + lane] : 0;
      __syncwarp();
      if (lane < rest) list[lane] = moved;
      have = rest;
      __syncwarp();
    }
  }
  drain(have);
  // the warps' sums in warp order
  if (warp > 0) {
#pragma unroll
    for (int pp = 0; pp < NP; ++pp)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float4*>(&sums[warp - 1][(pp * 2 + h) * 128 + lane * 4]) =
            make_float4(acc[pp][4 * h], acc[pp][4 * h + 1], acc[pp][4 * h + 2], acc[pp][4 * h + 3]);
  }
  __syncthreads();
  if (warp > 0) return;
  for (int w = 0; w < GRAD_WARPS - 1; ++w)
#pragma unroll
    for (int pp = 0; pp < NP; ++pp)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(&sums[w][(pp * 2 + h) * 128 + lane * 4]);
        acc[pp][4 * h] += v.x; acc[pp][4 * h + 1] += v.y; acc[pp][4 * h + 2] += v.z; acc[pp][4 * h + 3] += v.w;
      }
  store_row<NP>(p.dm + ((long long)n * p.E + e) * p.D, acc, pieces, lane);
}

}  // namespace

int launch_lmk_grad(const LmkGradArgs& a, cudaStream_t stream) {
  GradParams p;
  p.q = (const __nv_bfloat16*)a.lmk_q; p.m = (const __nv_bfloat16*)a.lmk_k; p.indices = a.indices; p.weights = a.weights;
  p.dw_rows = a.dw_rows; p.dw_all = a.dw_all; p.dq = (__nv_bfloat16*)a.dlmk_q; p.dm = (__nv_bfloat16*)a.dlmk_k;
  p.qbs = a.q_batch_stride; p.qrs = a.q_row_stride; p.mbs = a.k_batch_stride; p.mrs = a.k_row_stride;
  for (int i = 0; i < 3; ++i) { p.a_s[i] = a.dw_rows_stride[i]; p.b_s[i] = a.dw_all_stride[i]; }
  p.q_pos0 = a.q_pos0; p.N = a.N; p.Cq = a.Cq; p.E = a.E; p.D = a.D; p.K = a.K; p.rows_a = a.rows;
  p.scale = (float)(1.0 / sqrt((double)a.D));
  const long long blocks = (p.dm ? (long long)a.N * a.E : 0) + (p.dq ? ((long long)a.N * a.Cq + GRAD_WARPS - 1) / GRAD_WARPS : 0);
  if (blocks == 0) return 0;
  if (blocks >= (1ll << 31)) return GCA_ERR_TOO_LARGE;
  const unsigned grid = (unsigned)blocks;
  switch ((a.D + 255) / 256) {
    case 1: lmk_grad_kernel<1><<<grid, GRAD_WARPS * 32, 0, stream>>>(p); break;
    case 2: lmk_grad_kernel<2><<<grid, GRAD_WARPS * 32, 0, stream>>>(p); break;
    case 3: lmk_grad_kernel<3><<<grid, GRAD_WARPS * 32, 0, stream>>>(p); break;
    case 4: lmk_grad_kernel<4><<<grid, GRAD_WARPS * 32, 0, stream>>>(p); break;
    default: return GCA_ERR_SHAPE;
  }
  return (int)cudaGetLastError();
}

}  // namespace gca
