// out[m, :] = scale[m] * (x[m, :] . w^T) + residual[m, :] for a handful of rows (a decode step: one or two per sequence).
//
// Bound: latency.  768 x 768 weights are 1.2 MB, 0.2 us of HBM time; the 128 x 256-tile GEMM keeps 3 SMs busy with
// them for 9 us.  Here a block owns 8 or 16 output columns (96 blocks for 768), its 8 warps split the contraction, and every
// operand goes from global memory straight into mma.sync fragments: a 16-byte load per lane covers 8 consecutive k of one
// column (or row), and since a dot product does not care about the order of k, those 8 serve as the fragment's k slots
// of two steps -- the same permutation on both sides, no shared memory, no shuffles.  Partial sums of the warps are
// added in warp order.  With rms_eps the rows' mean squares are summed up from the same fragments, so that RMSNorm +
// projection (model/DRT.py:352-355, the gain folded into w) is one launch.  The weights are asked for (prefetch into L2)
// before the previous kernel on the stream has finished.
// One row, 768 -> 768: 9.3 -> 2.8 us.
#include "gca_common.cuh"

namespace gca {

namespace {

constexpr int WARPS = 8;

struct SkinnyParams {
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;
  __nv_bfloat16* out;
  const __nv_bfloat16* residual;   // or nullptr
  const float* row_scale;          // or nullptr
  long long x_stride, w_stride, out_stride, res_stride;
  int M, K;
  float rms_eps;                   // > 0: rows are scaled by 1 / rms(x) instead
};

__device__ __forceinline__ void mma_bf16(float c[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float sum_sq(const uint4& v, float s) {
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = __uint_as_float(w[i] << 16), b = __uint_as_float(w[i] & 0xffff0000u);
    s = fmaf(a, a, s);
    s = fmaf(b, b, s);
  }
  return s;
}

// A block: 16 MT rows x 8 NT columns.
template <int MT, int NT>
__global__ void __launch_bounds__(WARPS * 32)
skinny_linear_kernel(const SkinnyParams p) {
  constexpr int COLS = 8 * NT;
  __shared__ float part[WARPS][MT * 16][COLS];
  __shared__ float part_ss[WARPS][MT * 16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 2, quad = lane & 3;
  const int n0 = blockIdx.x * COLS, m0 = blockIdx.y * MT * 16, rows = min(MT * 16, p.M - m0), blocks = p.K / 32;
  const __nv_bfloat16* wrow = p.w + (long long)(n0 + grp) * p.w_stride + quad * 8;
  const __nv_bfloat16* x = p.x + m0 * p.x_stride + quad * 8;
  for (int kb = warp; kb < blocks; kb += WARPS)
#pragma unroll
    for (int t = 0; t < NT; ++t) asm volatile("prefetch.global.L2 [%0];" ::"l"(wrow + 8 * t * p.w_stride + kb * 32));
  pdl_trigger();
  pdl_wait();
  float acc[MT][NT][4], ss[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][t][i] = 0.f;
    ss[m][0] = ss[m][1] = 0.f;
  }
#pragma unroll 3
  for (int kb = warp; kb < blocks; kb += WARPS) {
    uint4 b[NT], a[MT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t) b[t] = *reinterpret_cast<const uint4*>(wrow + 8 * t * p.w_stride + kb * 32);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = m * 16 + h * 8 + grp;
        a[m][h] = r < rows ? *reinterpret_cast<const uint4*>(x + r * p.x_stride + kb * 32) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        mma_bf16(acc[m][t], a[m][0].x, a[m][1].x, a[m][0].y, a[m][1].y, b[t].x, b[t].y);
        mma_bf16(acc[m][t], a[m][0].z, a[m][1].z, a[m][0].w, a[m][1].w, b[t].z, b[t].w);
      }
      if (p.rms_eps > 0.f) {
        ss[m][0] = sum_sq(a[m][0], ss[m][0]);
        ss[m][1] = sum_sq(a[m][1], ss[m][1]);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = m * 16 + h * 8 + grp;
#pragma unroll
      for (int t = 0; t < NT; ++t)
        *reinterpret_cast<float2*>(&part[warp][r][t * 8 + quad * 2]) = make_float2(acc[m][t][2 * h], acc[m][t][2 * h + 1]);
      if (p.rms_eps > 0.f) {
        float s = ss[m][h];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (quad == 0) part_ss[warp][r] = s;
      }
    }
  __syncthreads();
  // a thread finishes two neighbouring columns of a row
  for (int i = threadIdx.x; i < rows * (COLS / 2); i += WARPS * 32) {
    const int r = i / (COLS / 2), c = (i % (COLS / 2)) * 2;
    const long long row = m0 + r;
    float2 t = make_float2(0.f, 0.f);
#pragma unroll
    for (int wv = 0; wv < WARPS; ++wv) {
      const float2 v = *reinterpret_cast<const float2*>(&part[wv][r][c]);
      t.x += v.x;
      t.y += v.y;
    }
    float sc = 1.f;
    if (p.rms_eps > 0.f) {
      float s = 0.f;
#pragma unroll
      for (int wv = 0; wv < WARPS; ++wv) s += part_ss[wv][r];
      sc = rsqrtf(s / (float)p.K + p.rms_eps);
    } else if (p.row_scale) sc = p.row_scale[row];
    float2 res = make_float2(0.f, 0.f);
    if (p.residual) {
      const unsigned v = *reinterpret_cast<const unsigned*>(p.residual + row * p.res_stride + n0 + c);
      res = make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    }
    const __nv_bfloat162 o = __floats2bfloat162_rn(fmaf(t.x, sc, res.x), fmaf(t.y, sc, res.y));
    *reinterpret_cast<__nv_bfloat162*>(p.out + row * p.out_stride + n0 + c) = o;
  }
}

}  // namespace

// Which products: what grows with rows and columns is the number of blocks, each of which reads its rows and its columns again, while
// the 128-row tiles of the tensor cores take the same ~5-7 us whatever the rows (~10 at 8,192 columns and few rows).  The line is where
// a wave of blocks is full: three per SM of 32 x 16, 14 per SM of 16 x 8 (which only read weights, once).  us, this form / tiles:
//   M = 16: 768 -> 4,096 3.5 / 6.1, 1,024 -> 8,192 7.4 / 9.7, 768 -> 16,384 (2,048 blocks) 9.3 / 9.2, 768 -> 50,304 24.5 / 19.5
//   M = 32: 768 -> 4,096 4.7 / 5.8, 1,024 -> 8,192 (512 blocks) 10.0 / 9.0, M = 17: 9.0 / 9.7; 768 -> 16,384 11.0 / 9.2
//   M = 64: 1,024 -> 3,072 (384 blocks) 5.5 / 6.1, 768 -> 4,096 (512) 8.0 / 5.5;  M = 96: 768 -> 2,304 (432) 4.9 / 5.4, 1,024 -> 3,072 9.9 / 6.2
//   M = 128: 768 -> 768 4.3 / 5.1, 768 -> 2,304 (576) 8.0 / 5.6, 768 -> 4,096 11.8 / 5.8
// With the norm the tiles cost a launch more, and the blocks' work per wave decides: 768 -> 2,304, M = 128: 8.7 / 8.9, 768 -> 4,096, M = 64:
// 8.7 / 8.8, 1,024 -> 3,072, M = 96: 10.4 / 8.5, 1,024 -> 4,096, M = 64: 10.4 / 9.3, 768 -> 4,096, M = 128: 12.8 / 9.1.
bool few_rows(long long M, int N, int K, bool with_norm, int sms) {
  if (M > GCA_SKINNY_ROWS) return false;
  if (M <= 16) return N / 8 <= 14 * sms;
  const long long blocks = N / 16 * ((M + 31) / 32);
  if (M <= 32) return blocks <= 4 * sms;
  return with_norm ? blocks * K <= 3ll * sms * 1024 : blocks <= 3 * sms;
}

// One block of rows (batches back to back), M <= GCA_SKINNY_ROWS.
int launch_skinny_linear(const LinearArgs& a, float rms_eps, cudaStream_t stream) {
  SkinnyParams p;
  p.x = (const __nv_bfloat16*)a.x; p.w = (const __nv_bfloat16*)a.w; p.out = (__nv_bfloat16*)a.out;
  p.residual = (const __nv_bfloat16*)a.residual; p.row_scale = a.row_scale;
  p.x_stride = a.x_stride; p.w_stride = a.w_stride; p.out_stride = a.out_stride; p.res_stride = a.residual_stride;
  p.M = (int)a.M; p.K = a.K; p.rms_eps = rms_eps;
  // more rows: 32 x 16 per block, so that neither operand is read by more blocks than needed to fill the SMs
  if (a.M <= 16) return (int)launch_dependent(skinny_linear_kernel<1, 1>, dim3((unsigned)(a.N / 8)), dim3(WARPS * 32), 0, stream, p);
  return (int)launch_dependent(skinny_linear_kernel<2, 2>, dim3((unsigned)(a.N / 16), (unsigned)((a.M + 31) / 32)), dim3(WARPS * 32), 0, stream, p);
}

}  // namespace gca
