// The GCA sub-layer of a decode step as ONE launch, for a handful of sequences: RMSNorm -> q projection -> attention over the
// retrieved chunks -> output projection (+ residual), model/DRT.py:345-394.
//
// Bound: latency.  For one sequence of a 768-wide model the step reads 4 MB; as three launches (projection, attention, projection)
// it takes ~6 us of launch calls on the host and three trips through global memory on the device.  Here a cluster of 16 CTAs has a
// sequence: its CTAs compute 1/16 of q's columns each, then 1/16 of the (head, slot) tiles, then 1/16 of the output's columns,
// and what one step leaves for the next stays in shared memory, read by the others through the cluster.  Everything that
// does not depend on the step before is asked for early: the K / V tiles (cp.async) while q is being computed, the output
// weights (registers) before the first cluster barrier.  16 SMs take ~50 bytes a clock each, 2.5 us for those 4 MB; wider
// grids would need grid-wide barriers, at more than a microsecond each.
// One sequence, 12 heads, K = 8: 13.1 -> 8.4 us per call (8.4 on the device, of which 4.8 are launch, barriers and hand-overs, 8.2 on
// the host); seven sequences 15 -> 9.
#include "gca_common.cuh"
#include "per_device.cuh"
#include "sm100_ptx.cuh"

namespace gca {

namespace {

using namespace sm100;

constexpr int CL = 16, WARPS = 16, THREADS = WARPS * 32;   // CTAs of a cluster; warps of a CTA
constexpr int TILE = 64 * 64 * 2;                          // one K or V tile
constexpr int MAX_UNITS = 12;                              // (head, slot) tiles of a CTA, 16 KB of shared memory each

struct LayerParams {
  const __nv_bfloat16* x;
  const __nv_bfloat16* wq;
  const __nv_bfloat16* wo;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  const int32_t* indices;
  const float* weights;
  const __nv_bfloat16* residual;   // or nullptr
  __nv_bfloat16* out;
  int32_t* status;
  long long wq_stride, wo_stride, ks[4], vs[4], res_batch, res_row;
  int H, G, K, C, units;           // units: (head, slot) tiles of a CTA
  float eps, c2;                   // c2: softmax scale in base 2
};

// Products go through mma.sync with the weights (or K rows) as the 16-row operand and the one or two query rows as two of the eight
// columns.  A 16-byte piece per lane covers eight consecutive k of one row; a dot product does not care about the order of k,
// so those eight serve as the fragments' k slots of two steps, the same on both sides.
__device__ __forceinline__ void mma_piece(float c[4], const uint4& row, const uint4& row8, const uint4& b) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(row.x), "r"(row8.x), "r"(row.y), "r"(row8.y), "r"(b.x), "r"(b.y));
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(row.z), "r"(row8.z), "r"(row.w), "r"(row8.w), "r"(b.z), "r"(b.w));
}
__device__ __forceinline__ void unpack8(const uint4& v, float f[8]) {
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// A word of another CTA's shared memory, at the address the same variable has here.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(cta));
  return r;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_cluster_16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// A CTA's 16 HQ columns of a projection: this warp's share of the contraction, blocks of 32 k (warp, warp + 16).
template <int HQ>
struct Share {
  static constexpr int BLOCKS = 8 * HQ, N = (BLOCKS + WARPS - 1) / WARPS;
  uint4 w[N][HQ][2];
};
template <int HQ>
__device__ __forceinline__ void load_weights(Share<HQ>& f, const __nv_bfloat16* w, long long stride, int warp, int lane) {
#pragma unroll
  for (int b = 0; b < Share<HQ>::N; ++b)
    if (warp + b * WARPS < Share<HQ>::BLOCKS)
#pragma unroll
      for (int t = 0; t < HQ; ++t)
#pragma unroll
        for (int r = 0; r < 2; ++r)
          f.w[b][t][r] = *reinterpret_cast<const uint4*>(w + (t * 16 + r * 8 + (lane >> 2)) * stride + (warp + b * WARPS) * 32 + (lane & 3) * 8);
}
// part[warp][column][s] = this warp's share of the dot products; x: the query rows' pieces (zero in lanes of other columns)
template <int HQ, int S>
__device__ __forceinline__ void project(const Share<HQ>& f, const uint4* x, float (*part)[16 * HQ][S], int warp, int lane) {
#pragma unroll
  for (int t = 0; t < HQ; ++t) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int b = 0; b < Share<HQ>::N; ++b)
      if (warp + b * WARPS < Share<HQ>::BLOCKS) mma_piece(c, f.w[b][t][0], f.w[b][t][1], x[b]);
    if ((lane & 3) == 0)
#pragma unroll
      for (int s = 0; s < S; ++s) {
        part[warp][t * 16 + (lane >> 2)][s] = c[s];
        part[warp][t * 16 + 8 + (lane >> 2)][s] = c[2 + s];
      }
  }
}
template <int HQ, int S>
__device__ __forceinline__ float sum_shares(const float (*part)[16 * HQ][S], int col, int s) {
  float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < WARPS; ++i) v[i & 3] += part[i][col][s];
  return (v[0] + v[1]) + (v[2] + v[3]);
}

// HQ = heads / 4.  S: query rows (1 or 2).
template <int HQ, int S>
__global__ void __launch_bounds__(THREADS, 1)
layer_decode_kernel(const __grid_constant__ LayerParams p) {
  constexpr int DIM = HQ * 256, COLS = DIM / CL;           // columns of a CTA: 16 HQ
  extern __shared__ __align__(128) uint8_t tiles[];        // [units][K | V]: row r's piece c lies at piece c ^ 4 (r & 1)
  __shared__ float part[WARPS][COLS][S], part_ss[WARPS][S];
  __shared__ __align__(16) __nv_bfloat16 q_mine[S][COLS];
  __shared__ __align__(16) float half_o[2 * MAX_UNITS][S][64], half_m[2 * MAX_UNITS][S], half_l[2 * MAX_UNITS][S];
  __shared__ float factor[2 * MAX_UNITS][S];               // weight of a half tile in its head's output
  __shared__ float head_o[MAX_UNITS][S][64];               // sum over this CTA's slots of the i-th head it has a part of
  __shared__ __align__(16) __nv_bfloat16 attn[S][DIM];
  __shared__ float unit_w[MAX_UNITS];
  __shared__ int unit_chunk[MAX_UNITS], unit_head[MAX_UNITS];
  __shared__ int first_cta[4 * HQ], last_cta[4 * HQ], first_head[CL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cta = (int)cluster_rank(), n = blockIdx.x / CL;
  const int total = p.H * p.K, u0 = min(cta * p.units, total), nu = min(p.units, total - u0);
  const __nv_bfloat16* wq = p.wq + cta * COLS * p.wq_stride;
  const __nv_bfloat16* wo = p.wo + cta * COLS * p.wo_stride;
  if (threadIdx.x < nu) unit_head[threadIdx.x] = (u0 + threadIdx.x) / p.K;
  else if (threadIdx.x >= 64 && threadIdx.x < 64 + 4 * HQ) {
    const int h = threadIdx.x - 64;
    first_cta[h] = h * p.K / p.units;
    last_cta[h] = ((h + 1) * p.K - 1) / p.units;
  } else if (threadIdx.x >= 128 && threadIdx.x < 128 + CL) first_head[threadIdx.x - 128] = (threadIdx.x - 128) * p.units / p.K;
  const int slot = threadIdx.x < nu ? (u0 + threadIdx.x) % p.K : 0;
  // 128-byte lines of the output weights into L2
  for (int i = threadIdx.x; i < COLS * 4 * HQ; i += THREADS)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(wo + (i / (4 * HQ)) * p.wo_stride + i % (4 * HQ) * 64));
  pdl_trigger();
  pdl_wait();
  // ---- q: everything it needs in flight, then the K / V tiles behind it
  Share<HQ> f;
  uint4 x[Share<HQ>::N];
  if (threadIdx.x < nu) {
    const int id = p.indices[n * p.K + slot];
    const float w = p.weights[n * p.K + slot];
    const bool valid = id >= 0 && id < p.C;
    if (id >= p.C && p.status) atomicOr(p.status, GCA_STATUS_BAD_INDEX);
    unit_chunk[threadIdx.x] = valid ? id : -1;
    unit_w[threadIdx.x] = w;
  }
  load_weights<HQ>(f, wq, p.wq_stride, warp, lane);
#pragma unroll
  for (int b = 0; b < Share<HQ>::N; ++b) {
    x[b] = make_uint4(0, 0, 0, 0);
    if ((lane >> 2) < S && warp + b * WARPS < Share<HQ>::BLOCKS)
      x[b] = *reinterpret_cast<const uint4*>(p.x + ((long long)n * S + (lane >> 2)) * DIM + (warp + b * WARPS) * 32 + (lane & 3) * 8);
  }
  __syncthreads();
  for (int u = 0; u < nu; ++u) {
    const int c = unit_chunk[u];
    if (c < 0) continue;
    const int h = unit_head[u] / p.G, row = threadIdx.x >> 3, piece = threadIdx.x & 7;
    uint8_t* dst = tiles + u * 2 * TILE + row * 128 + ((piece ^ ((row & 1) << 2)) << 4);
    cp_async16(dst, p.k + n * p.ks[0] + c * p.ks[1] + row * p.ks[2] + h * p.ks[3] + piece * 8);
    cp_async16(dst + TILE, p.v + n * p.vs[0] + c * p.vs[1] + row * p.vs[2] + h * p.vs[3] + piece * 8);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  project<HQ, S>(f, x, part, warp, lane);
  {
    float ss = 0.f;
#pragma unroll
    for (int b = 0; b < Share<HQ>::N; ++b) {
      float v[8];
      unpack8(x[b], v);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
    }
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    ss += __shfl_xor_sync(0xffffffffu, ss, 2);
    if ((lane & 3) == 0 && (lane >> 2) < S) part_ss[warp][lane >> 2] = ss;
  }
  load_weights<HQ>(f, wo, p.wo_stride, warp, lane);        // used two barriers later
  __syncthreads();
  if (threadIdx.x < COLS * S) {
    const int s = threadIdx.x / COLS, col = threadIdx.x % COLS;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) ss += part_ss[i][s];
    q_mine[s][col] = __float2bfloat16_rn(sum_shares<HQ, S>(part, col, s) * rsqrtf(ss * (1.0f / DIM) + p.eps));
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  cluster_sync();

  // ---- attention: a warp takes 32 keys of a tile
  const int grp = lane >> 2, quad = lane & 3, vgrp = lane >> 3, piece = lane & 7;
  for (int hu = warp; hu < 2 * nu; hu += WARPS) {
    const int u = hu >> 1, h = unit_head[u];
    const uint8_t* kt = tiles + u * 2 * TILE + (hu & 1) * (TILE / 2);
    if (unit_chunk[u] < 0) continue;
    uint4 qv[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
    if (grp < S)
#pragma unroll
      for (int j = 0; j < 2; ++j) {                        // a piece of q lies in one CTA
        const int col = h * 64 + (quad + 4 * j) * 8;
        qv[j] = ld_cluster_16(cluster_addr(&q_mine[grp][col % COLS], col / COLS));
      }
    // scores: rows grp and grp + 8 of two 16-key blocks; lanes with quad = 0 hold query rows 0 and 1
    float c[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint8_t* src = kt + (t * 16 + grp) * 128 + (((quad + 4 * j) ^ ((grp & 1) << 2)) << 4);
        mma_piece(c[t], *reinterpret_cast<const uint4*>(src), *reinterpret_cast<const uint4*>(src + 8 * 128), qv[j]);
      }
    }
    float o[S][8], l[S], m[S], e[S][4];
#pragma unroll
    for (int s = 0; s < S; ++s) {                          // e[s][i]: key 8 i + grp
#pragma unroll
      for (int i = 0; i < 4; ++i) e[s][i] = c[i >> 1][(i & 1) * 2 + s] * p.c2;
      m[s] = fmaxf(fmaxf(e[s][0], e[s][1]), fmaxf(e[s][2], e[s][3]));
#pragma unroll
      for (int of = 4; of < 32; of <<= 1) m[s] = fmaxf(m[s], __shfl_xor_sync(0xffffffffu, m[s], of));
#pragma unroll
      for (int i = 0; i < 4; ++i) e[s][i] = ex2_approx(e[s][i] - m[s]);
      l[s] = (e[s][0] + e[s][1]) + (e[s][2] + e[s][3]);
#pragma unroll
      for (int of = 4; of < 32; of <<= 1) l[s] += __shfl_xor_sync(0xffffffffu, l[s], of);
#pragma unroll
      for (int d = 0; d < 8; ++d) o[s][d] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {                          // V row 4 i + vgrp, eight columns per lane
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(kt + TILE + (4 * i + vgrp) * 128 + ((piece ^ ((vgrp & 1) << 2)) << 4)), v);
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const float w = __shfl_sync(0xffffffffu, e[s][i >> 1], ((i & 1) * 4 + vgrp) * 4);
#pragma unroll
        for (int d = 0; d < 8; ++d) o[s][d] = fmaf(w, v[d], o[s][d]);
      }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
#pragma unroll
      for (int d = 0; d < 8; ++d) {
        o[s][d] += __shfl_xor_sync(0xffffffffu, o[s][d], 8);
        o[s][d] += __shfl_xor_sync(0xffffffffu, o[s][d], 16);
      }
      if (vgrp == 0) {
        *reinterpret_cast<float4*>(&half_o[hu][s][piece * 8]) = make_float4(o[s][0], o[s][1], o[s][2], o[s][3]);
        *reinterpret_cast<float4*>(&half_o[hu][s][piece * 8 + 4]) = make_float4(o[s][4], o[s][5], o[s][6], o[s][7]);
      }
      if (lane == 0) { half_m[hu][s] = m[s]; half_l[hu][s] = l[s]; }
    }
  }
  __syncthreads();
  if (threadIdx.x < nu * S) {                              // the two halves of every tile, and the slot's weight
    const int u = threadIdx.x / S, s = threadIdx.x % S;
    if (unit_chunk[u] >= 0) {
      const float ma = half_m[2 * u][s], mb = half_m[2 * u + 1][s], mm = fmaxf(ma, mb);
      const float ea = ex2_approx(ma - mm), eb = ex2_approx(mb - mm);
      const float w = unit_w[u] / (ea * half_l[2 * u][s] + eb * half_l[2 * u + 1][s]);
      factor[2 * u][s] = w * ea;
      factor[2 * u + 1][s] = w * eb;
    }
  }
  __syncthreads();
  const int h_first = first_head[cta], parts = nu > 0 ? unit_head[nu - 1] - h_first + 1 : 0;
  for (int t = threadIdx.x; t < parts * S * 64; t += THREADS) {      // this CTA's slots of a head, in slot order
    const int d = t & 63, s = (t >> 6) % S, h = h_first + (t >> 6) / S;
    const int lo = max(h * p.K, u0) - u0, hi = min((h + 1) * p.K, u0 + nu) - u0;
    float sum = 0.f;
    for (int u = lo; u < hi; ++u)
      if (unit_chunk[u] >= 0) sum += factor[2 * u][s] * half_o[2 * u][s][d] + factor[2 * u + 1][s] * half_o[2 * u + 1][s][d];
    head_o[h - h_first][s][d] = sum;
  }
  __syncwarp();
  cluster_sync();
  // ---- the whole attention row: the parts of every head, from the CTAs that have them
  for (int t = threadIdx.x; t < S * DIM; t += THREADS) {
    const int s = t / DIM, col = t % DIM, h = col >> 6, last = last_cta[h];
    float sum = 0.f;
    for (int c = first_cta[h]; c <= last; ++c) sum += ld_cluster_f32(cluster_addr(&head_o[h - first_head[c]][s][col & 63], c));
    attn[s][col] = __float2bfloat16_rn(sum);
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // done with the others' memory
  __syncthreads();
  // ---- output projection
#pragma unroll
  for (int b = 0; b < Share<HQ>::N; ++b) {
    x[b] = make_uint4(0, 0, 0, 0);
    if (grp < S && warp + b * WARPS < Share<HQ>::BLOCKS)
      x[b] = *reinterpret_cast<const uint4*>(&attn[grp][(warp + b * WARPS) * 32 + quad * 8]);
  }
  project<HQ, S>(f, x, part, warp, lane);
  __syncthreads();
  if (threadIdx.x < COLS * S) {
    const int s = threadIdx.x / COLS, col = cta * COLS + threadIdx.x % COLS;
    float v = sum_shares<HQ, S>(part, threadIdx.x % COLS, s);
    if (p.residual) v += __bfloat162float(p.residual[n * p.res_batch + s * p.res_row + col]);
    p.out[((long long)n * S + s) * DIM + col] = __float2bfloat16_rn(v);
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // nobody reads this CTA's memory any more
}

template <int HQ, int S>
int launch(const LayerDecodeArgs& a, const LayerParams& p, int dev, cudaStream_t stream) {
  auto kernel = layer_decode_kernel<HQ, S>;
  const size_t smem = (size_t)p.units * 2 * TILE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.N * CL)); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CL; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  // How many clusters of the largest CTA run at a time (each needs 16 SMs of one GPC), and the two limits raised: a device's own, so
  // once per device.  If that fails the call takes three launches, and the next one tries again.
  static PerDevice clusters;
  int most = 0;
  const bool known = clusters.get(dev, &most, [&](int* n) {
    cudaLaunchConfig_t largest = cfg;
    largest.dynamicSmemBytes = MAX_UNITS * 2 * TILE;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_UNITS * 2 * TILE) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(n, kernel, &largest) == cudaSuccess)
      return true;
    cudaGetLastError();
    return false;
  });
  if (!known || a.N > most) return GCA_ERR_ALGO;
  return (int)cudaLaunchKernelEx(&cfg, kernel, p);
}

template <int S>
int launch_heads(const LayerDecodeArgs& a, const LayerParams& p, int dev, cudaStream_t stream) {
  switch (a.H) {
    case 4: return launch<1, S>(a, p, dev, stream);
    case 8: return launch<2, S>(a, p, dev, stream);
    case 12: return launch<3, S>(a, p, dev, stream);
    default: return launch<4, S>(a, p, dev, stream);
  }
}

}  // namespace

// As many sequences as clusters run at a time, 7 on a B200 (a second wave takes longer than three launches: 16.9 against 14.4 us), 4, 8,
// 12 or 16 heads, and no more (head, slot) tiles per CTA than fit into its shared memory; anything else is GCA_ERR_ALGO, before
// anything has been launched: more sequences fill the chip as three launches.  `dev`: the current device.
int launch_layer_decode(const LayerDecodeArgs& a, int dev, cudaStream_t stream) {
  LayerParams p;
  p.units = (a.H * a.K + CL - 1) / CL;
  if (a.S < 1 || a.S > 2 || a.H % 4 != 0 || a.H < 4 || a.H > 16 || p.units > MAX_UNITS) return GCA_ERR_ALGO;
  p.x = (const __nv_bfloat16*)a.x; p.wq = (const __nv_bfloat16*)a.wq; p.wo = (const __nv_bfloat16*)a.wo;
  p.k = (const __nv_bfloat16*)a.k_cache; p.v = (const __nv_bfloat16*)a.v_cache; p.indices = a.indices; p.weights = a.weights;
  p.residual = (const __nv_bfloat16*)a.residual; p.out = (__nv_bfloat16*)a.out; p.status = a.status;
  p.wq_stride = a.wq_stride; p.wo_stride = a.wo_stride; p.res_batch = a.residual_batch_stride; p.res_row = a.residual_stride;
  for (int i = 0; i < 4; ++i) { p.ks[i] = a.k_stride[i]; p.vs[i] = a.v_stride[i]; }
  p.H = a.H; p.G = a.H / a.Hkv; p.K = a.K; p.C = a.C; p.eps = a.eps; p.c2 = a.sm_scale * GCA_LOG2E;
  return a.S == 1 ? launch_heads<1>(a, p, dev, stream) : launch_heads<2>(a, p, dev, stream);
}

}  // namespace gca
