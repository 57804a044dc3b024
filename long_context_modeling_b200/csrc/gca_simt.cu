// CUDA-core GCA kernels with float32 arithmetic throughout.  They serve what the tensor-core kernels do not take (fewer than 64 query
// rows) and callers that ask for them; float32 with 64 rows goes to gca_f32_sm100.cu, which is faster and closer to 64 bits.  One block of four
// warps owns one (sequence, query chunk, head) in the q-major kernels and one (sequence, cache chunk, kv head) in the
// kv-major backward kernel, so no atomics are needed and results are bit-reproducible.
//
// Bound: the FMA pipe (73 TFLOP/s measured on this part; the packed form is no faster).  A product of two 64 x 64
// tiles is 64 steps of 64 x 64 FMA, so what matters is how few other instructions go with them: a warp owns 16
// rows x 64 columns of every product, a thread 4 x 8, which is 12 16-byte shared loads per 128 FMA (a 4 x 4 tile with scalar
// loads: 64 per 128).  A warp owns whole rows, so the softmax stays inside it, and the rows it writes as the A
// operand of the next product are read by nobody else: blocks synchronise only for the K / V (Q / dO) tiles,
// which cp.async brings in one step ahead.  The kv-major kernel works on TRANSPOSED scores (rows = keys) for the same
// reason; what it needs per query row, Di = rowsum(P dP), comes from the q-major kernel.
// 2 x 64 chunks x 12 heads, top-8, float32: forward 477 -> 355 us, q-major 689 -> 481 us, kv-major 1031 -> 588 us (785 when its
// blocks started in table order head by head, the longest units of the last head almost at the end).
#include "gca_simt.cuh"

namespace gca {

namespace {

template <typename E>
__global__ void __launch_bounds__(NTHREADS, 4)
fwd_simt_kernel(const E* __restrict__ q, const E* __restrict__ kc, const E* __restrict__ vc,
                const int32_t* __restrict__ indices, const float* __restrict__ weights,
                E* __restrict__ out, float* __restrict__ lse, int32_t* status, Geom g) {
  extern __shared__ __align__(16) float smem[];
  fwd_unit<E>(smem, blockIdx.x, blockIdx.y, q, kc, vc, indices, weights, out, lse, status, g);
}

template <typename E>
__global__ void __launch_bounds__(NTHREADS, 2)
bwd_q_simt_kernel(const E* __restrict__ q, const E* __restrict__ kc, const E* __restrict__ vc,
                  const int32_t* __restrict__ indices, const float* __restrict__ weights,
                  const E* __restrict__ dout, const float* __restrict__ lse, E* __restrict__ dq,
                  float* __restrict__ dw_part, float* __restrict__ row_di, Geom g,
                  long long dos0, long long dos1, long long dos2, long long dos3) {
  extern __shared__ __align__(16) float smem[];
  bwd_q_unit<E, 1>(smem, blockIdx.x, blockIdx.y, q, kc, vc, indices, weights, dout, lse, dq, dw_part, row_di, g, dos0, dos1, dos2, dos3);
}

template <typename E>
__global__ void __launch_bounds__(NTHREADS, 2)
bwd_kv_simt_kernel(const E* __restrict__ q, const E* __restrict__ kc, const E* __restrict__ vc,
                   const float* __restrict__ weights, const E* __restrict__ dout, const float* __restrict__ lse,
                   const float* __restrict__ row_di, E* __restrict__ dk, E* __restrict__ dv, Csr csr, Geom g,
                   long long dos0, long long dos1, long long dos2, long long dos3,
                   long long dks0, long long dks1, long long dks2, long long dks3,
                   long long dvs0, long long dvs1, long long dvs2, long long dvs3) {
  extern __shared__ __align__(16) float smem[];
  bwd_kv_unit<E>(smem, csr.unit_tab[blockIdx.x / g.Hkv], blockIdx.x % g.Hkv, q, kc, vc, weights, dout, lse, row_di, dk, dv, csr, g, dos0, dos1, dos2, dos3,
                 dks0, dks1, dks2, dks3, dvs0, dvs1, dvs2, dvs3);
}

// One thread per (row block, slot), whatever the order of the loads the same order of the sum.  Four heads' loads are in flight at a
// time: one by one they cost 10 us for 12 heads x 4 partials, whatever the number of rows.
template <int PARTS>
__global__ void dw_reduce_kernel(const float* __restrict__ part, float* __restrict__ dw, int ZJ, int Hq, int K) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)ZJ * K) return;
  const long long zj = i / K;
  const float* p = part + (zj * Hq * K + (i - zj * K)) * PARTS;
  float t = 0.f;
#pragma unroll 4
  for (int h = 0; h < Hq; ++h, p += K * PARTS) {
    if (PARTS == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p));
      t += v.x; t += v.y; t += v.z; t += v.w;
    } else {
      t += __ldg(p);
    }
  }
  dw[i] = t;
}

template <typename E>
int fwd_simt_typed(const GcaFwdArgs& a, cudaStream_t stream) {
  const size_t smem = FWD_UNIT_SMEM;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(fwd_simt_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((unsigned)(a.N * a.J), (unsigned)a.Hq);
  fwd_simt_kernel<E><<<grid, NTHREADS, smem, stream>>>((const E*)a.q, (const E*)a.k_cache, (const E*)a.v_cache,
                                                       a.indices, a.weights, (E*)a.out, a.lse, a.status, make_geom(a));
  return (int)cudaGetLastError();
}

template <typename E>
int bwd_simt_typed(const GcaBwdArgs& a, const Csr& csr, float* dw_part, float* row_di, cudaStream_t stream, unsigned stages) {
  const Geom g = make_geom(a);
  if (stages & GCA_BWD_STAGE_Q) {
    GCA_CUDA_CHECK(cudaFuncSetAttribute(bwd_q_simt_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_Q_UNIT_SMEM));
    const dim3 grid((unsigned)(a.N * a.J), (unsigned)a.Hq);
    if (grid.x > 0)
      bwd_q_simt_kernel<E><<<grid, NTHREADS, BWD_Q_UNIT_SMEM, stream>>>(
          (const E*)a.q, (const E*)a.k_cache, (const E*)a.v_cache, a.indices, a.weights, (const E*)a.dout, a.lse,
          (E*)a.dq, dw_part, row_di, g, a.do_stride[0], a.do_stride[1], a.do_stride[2], a.do_stride[3]);
    GCA_CUDA_CHECK(cudaGetLastError());
  }
  if (stages & GCA_BWD_STAGE_KV) {
    GCA_CUDA_CHECK(cudaFuncSetAttribute(bwd_kv_simt_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_KV_UNIT_SMEM));
    const unsigned grid = (unsigned)((long long)a.N * a.C * a.Hkv);
    bwd_kv_simt_kernel<E><<<grid, NTHREADS, BWD_KV_UNIT_SMEM, stream>>>(
        (const E*)a.q, (const E*)a.k_cache, (const E*)a.v_cache, a.weights, (const E*)a.dout, a.lse, row_di,
        (E*)a.dk_cache, (E*)a.dv_cache, csr, g,
        a.do_stride[0], a.do_stride[1], a.do_stride[2], a.do_stride[3],
        a.dk_stride[0], a.dk_stride[1], a.dk_stride[2], a.dk_stride[3],
        a.dv_stride[0], a.dv_stride[1], a.dv_stride[2], a.dv_stride[3]);
    GCA_CUDA_CHECK(cudaGetLastError());
  }
  return 0;
}

}  // namespace

int launch_fwd_simt(const GcaFwdArgs& a, cudaStream_t stream) {
  if (a.dtype == GCA_BF16) return fwd_simt_typed<__nv_bfloat16>(a, stream);
  if (a.dtype == GCA_F32) return fwd_simt_typed<float>(a, stream);
  return GCA_ERR_DTYPE;
}

int launch_bwd_simt(const GcaBwdArgs& a, const Csr& csr, float* dw_part, float* row_di, cudaStream_t stream, unsigned stages) {
  if (a.dtype == GCA_BF16) return bwd_simt_typed<__nv_bfloat16>(a, csr, dw_part, row_di, stream, stages);
  if (a.dtype == GCA_F32) return bwd_simt_typed<float>(a, csr, dw_part, row_di, stream, stages);
  return GCA_ERR_DTYPE;
}

int launch_dw_reduce(const float* dw_part, float* dw, int ZJ, int Hq, int K, int parts, cudaStream_t stream) {
  const long long total = (long long)ZJ * K;
  if (total == 0) return 0;
  const unsigned blocks = (unsigned)((total + 63) / 64);
  if (parts == 4) dw_reduce_kernel<4><<<blocks, 64, 0, stream>>>(dw_part, dw, ZJ, Hq, K);
  else dw_reduce_kernel<1><<<blocks, 64, 0, stream>>>(dw_part, dw, ZJ, Hq, K);
  return (int)cudaGetLastError();
}

}  // namespace gca
