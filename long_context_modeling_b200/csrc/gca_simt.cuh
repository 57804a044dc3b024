// One unit of GCA with float32 multiply-adds throughout, by 128 threads: the body of the CUDA-core kernels (gca_simt.cu), and what the float32
// tensor-core kernels (gca_f32_sm100.cu) do with a unit that lies outside their range.
#pragma once
#include "gca_common.cuh"

namespace gca {

namespace {

constexpr int T = 64;            // tile edge (keys per chunk, head dim, max query rows)
constexpr int LD = T + 4;        // row pitch of operand tiles: eight rows of 16 bytes hit all banks once
constexpr int LDP = T + 8;       // row pitch of tiles written by (4 rows x 8 columns) lanes
constexpr int NTHREADS = 128;
constexpr int TILE = T * LD, TILE_P = T * LDP;

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// The block's first 128 threads, which are all that a unit takes.
__device__ __forceinline__ void unit_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory"); }

// A (rows x 64) tile whose rows are `row_stride` elements apart; rows past `rows` become zeros.  float32 arrives
// asynchronously (one commit group, taken by the caller), bf16 is widened on the way.
__device__ __forceinline__ void load_tile(float* dst, const float* src, long long row_stride, int rows) {
  for (int i = threadIdx.x; i < T * (T / 4); i += NTHREADS) {
    const int r = i >> 4, c = (i & 15) * 4;
    if (r < rows) cp_async16(dst + r * LD + c, src + r * row_stride + c);
    else *reinterpret_cast<float4*>(dst + r * LD + c) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
__device__ __forceinline__ void load_tile(float* dst, const __nv_bfloat16* src, long long row_stride, int rows) {
  for (int i = threadIdx.x; i < T * (T / 8); i += NTHREADS) {
    const int r = i >> 3, c = (i & 7) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < rows) v = *reinterpret_cast<const uint4*>(src + r * row_stride + c);
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float4*>(dst + r * LD + c + 4 * h) =
          make_float4(__uint_as_float(w[2 * h] << 16), __uint_as_float(w[2 * h] & 0xffff0000u), __uint_as_float(w[2 * h + 1] << 16),
                      __uint_as_float(w[2 * h + 1] & 0xffff0000u));
  }
}

// What a thread owns of a product: rows row0 + 4 i (i < 4) and columns tx + 8 j (NT products) or tx * 4 + 32 (j / 4) + j % 4 (NN).
struct Own {
  int row0, tx;
  __device__ __forceinline__ Own() {
    const int lane = threadIdx.x & 31;
    row0 = (threadIdx.x >> 5) * 16 + (lane >> 3);
    tx = lane & 7;
  }
};

// acc[i][j] = sum_d A[row_i][d] B[col_j][d]
__device__ __forceinline__ void mma_nt(const float* A, const float* B, const Own& o, float acc[4][8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  const float* a0 = A + o.row0 * LD;
  const float* b0 = B + o.tx * LD;
#pragma unroll 4
  for (int d = 0; d < T; d += 4) {
    float4 a[4], b[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + 4 * i * LD + d);
#pragma unroll
    for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(b0 + 8 * j * LD + d);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
      }
  }
}

// acc[i][j] += sum_r A[row_i][r] B[r][col_j]   (A: pitch LDP, this warp's own rows)
__device__ __forceinline__ void mma_nn_acc(const float* A, const float* B, const Own& o, float acc[4][8]) {
  const float* a0 = A + o.row0 * LDP;
  const float* b0 = B + o.tx * 4;
#pragma unroll 4
  for (int r = 0; r < T; r += 4) {
    float4 a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + 4 * i * LDP + r);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 b = *reinterpret_cast<const float4*>(b0 + (r + x) * LD), c = *reinterpret_cast<const float4*>(b0 + (r + x) * LD + 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float av = x == 0 ? a[i].x : x == 1 ? a[i].y : x == 2 ? a[i].z : a[i].w;
        acc[i][0] = fmaf(av, b.x, acc[i][0]); acc[i][1] = fmaf(av, b.y, acc[i][1]);
        acc[i][2] = fmaf(av, b.z, acc[i][2]); acc[i][3] = fmaf(av, b.w, acc[i][3]);
        acc[i][4] = fmaf(av, c.x, acc[i][4]); acc[i][5] = fmaf(av, c.y, acc[i][5]);
        acc[i][6] = fmaf(av, c.z, acc[i][6]); acc[i][7] = fmaf(av, c.w, acc[i][7]);
      }
    }
  }
}

// Write a thread's NT-shaped values as rows of the next product's A operand.
__device__ __forceinline__ void put_rows(float* P, const Own& o, const float v[4][8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) P[(o.row0 + 4 * i) * LDP + o.tx + 8 * j] = v[i][j];
}

__device__ __forceinline__ void store4(float* dst, const float* v, float s) {
  *reinterpret_cast<float4*>(dst) = make_float4(v[0] * s, v[1] * s, v[2] * s, v[3] * s);
}
__device__ __forceinline__ void store4(__nv_bfloat16* dst, const float* v, float s) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v[0] * s, v[1] * s), b = __floats2bfloat162_rn(v[2] * s, v[3] * s);
  *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}
template <typename E>
__device__ __forceinline__ void store_rows(E* base, long long row_stride, int rows, const Own& o, const float acc[4][8], float s) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = o.row0 + 4 * i;
    if (r >= rows) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) store4(base + r * row_stride + o.tx * 4 + 32 * h, &acc[i][4 * h], s);
  }
}

// Reduce over the 8 lanes that share a row.
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
  for (int of = 4; of > 0; of >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, of));
  return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int of = 4; of > 0; of >>= 1) v += __shfl_xor_sync(0xffffffffu, v, of);
  return v;
}

// The next slot from k on that reads a chunk (K if none).
__device__ __forceinline__ int next_slot(const int32_t* indices, long long zj, const Geom& g, int k, int& idx) {
  for (; k < g.K; ++k) {
    idx = slot_chunk(indices, zj, g.K, k);
    if (idx >= 0 && idx < g.C) break;
  }
  return k;
}

// ------------------------------------------------------------------------------------
// forward: one (row block zj, head)
// ------------------------------------------------------------------------------------
constexpr int FWD_UNIT_SMEM = (2 * TILE + TILE_P) * sizeof(float);
template <typename E>
__device__ __forceinline__ void fwd_unit(float* smem, int zj, int h, const E* __restrict__ q, const E* __restrict__ kc, const E* __restrict__ vc,
                                         const int32_t* __restrict__ indices, const float* __restrict__ weights,
                                         E* __restrict__ out, float* __restrict__ lse, int32_t* status, const Geom& g) {
  float *sQ = smem, *sV = sQ + TILE, *sK = sV + TILE, *sP = sK;      // P takes K's place: four blocks fit on an SM
  const int n = zj / g.J, j = zj % g.J, hk = h / g.G;
  const Own own;
  // padding slots and ids outside the cache
  for (int k = 0; k < g.K; ++k) {
    const int idx = slot_chunk(indices, zj, g.K, k);
    if (idx >= 0 && idx < g.C) continue;
    if (idx >= g.C && status && threadIdx.x == 0) atomicOr(status, GCA_STATUS_BAD_INDEX);
    if (lse) for (int r = threadIdx.x; r < g.S; r += NTHREADS) lse[(((long long)zj * g.Hq + h) * g.K + k) * g.S + r] = 0.f;
  }
  auto k_tile = [&](int idx) { load_tile(sK, kc + n * g.ks[0] + idx * g.ks[1] + hk * g.ks[3], g.ks[2], T); };
  auto v_tile = [&](int idx) { load_tile(sV, vc + n * g.vs[0] + idx * g.vs[1] + hk * g.vs[3], g.vs[2], T); };
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[i][b] = 0.f;
  const float c2 = g.sm_scale * GCA_LOG2E;

  int idx = -1, k = next_slot(indices, zj, g, 0, idx);
  if (k < g.K) {
    load_tile(sQ, q + n * g.qs[0] + j * g.qs[1] + h * g.qs[2], g.qs[3], g.S);
    k_tile(idx);
    cp_commit();
    v_tile(idx);
    cp_commit();
  }
  while (k < g.K) {
    int idx_next = -1;
    const int k_next = next_slot(indices, zj, g, k + 1, idx_next);
    const float w = weights[(long long)zj * g.K + k];
    cp_wait<1>();                              // Q and K are here, V may still be on its way
    unit_sync();
    float s[4][8];
    mma_nt(sQ, sK, own, s);
    unit_sync();                           // every warp is done with K
    float* lse_row = lse ? lse + (((long long)zj * g.Hq + h) * g.K + k) * g.S : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float m = -INFINITY;
#pragma unroll
      for (int b = 0; b < 8; ++b) { s[i][b] *= c2; m = fmaxf(m, s[i][b]); }
      m = row_max(m);
      if (g.off_by_one > 0.f) m = fmaxf(m, 0.f);
      float l = 0.f;
#pragma unroll
      for (int b = 0; b < 8; ++b) { s[i][b] = exp2f(s[i][b] - m); l += s[i][b]; }
      l = row_sum(l);
      if (g.off_by_one > 0.f) l += g.off_by_one * exp2f(-m);
      const int r = own.row0 + 4 * i;
      if (lse_row && own.tx == 0 && r < g.S) lse_row[r] = m + log2f(l);
      const float f = w / l;
#pragma unroll
      for (int b = 0; b < 8; ++b) s[i][b] *= f;
    }
    put_rows(sP, own, s);
    cp_wait<0>();                              // V is here
    unit_sync();
    mma_nn_acc(sP, sV, own, acc);
    unit_sync();                           // every warp is done with P and V
    if (k_next < g.K) {
      k_tile(idx_next);
      cp_commit();
      v_tile(idx_next);
      cp_commit();
    }
    k = k_next;
    idx = idx_next;
  }
  store_rows(out + n * g.os[0] + j * g.os[1] + h * g.os[2], g.os[3], g.S, own, acc, 1.0f);
}

// ------------------------------------------------------------------------------------
// backward, q-major: one (sequence, query chunk, q head): dQ, the per-head part of dw (PARTS = 4: of every warp's rows), and Di = rowsum(P dP) of
// every (row, slot) for the kv-major unit.
// ------------------------------------------------------------------------------------
constexpr int BWD_Q_UNIT_SMEM = (4 * TILE + TILE_P + 2 * (NTHREADS / 32)) * sizeof(float);
template <typename E, int PARTS>
__device__ __forceinline__ void bwd_q_unit(float* smem, int zj, int h, const E* __restrict__ q, const E* __restrict__ kc, const E* __restrict__ vc,
                                           const int32_t* __restrict__ indices, const float* __restrict__ weights,
                                           const E* __restrict__ dout, const float* __restrict__ lse, E* __restrict__ dq,
                                           float* __restrict__ dw_part, float* __restrict__ row_di, const Geom& g,
                                           long long dos0, long long dos1, long long dos2, long long dos3) {
  float *sQ = smem, *sdO = sQ + TILE, *sK = sdO + TILE, *sV = sK + TILE, *sdS = sV + TILE;
  float (*red)[NTHREADS / 32] = reinterpret_cast<float (*)[NTHREADS / 32]>(sdS + TILE_P);
  const int n = zj / g.J, j = zj % g.J, hk = h / g.G;
  const Own own;
  const float c2 = g.sm_scale * GCA_LOG2E;
  for (int k = threadIdx.x; k < g.K; k += NTHREADS) {
    const int idx = slot_chunk(indices, zj, g.K, k);
    if (idx < 0 || idx >= g.C)
      for (int x = 0; x < PARTS; ++x) dw_part[(((long long)zj * g.Hq + h) * g.K + k) * PARTS + x] = 0.f;
  }
  auto k_tile = [&](int idx) { load_tile(sK, kc + n * g.ks[0] + idx * g.ks[1] + hk * g.ks[3], g.ks[2], T); };
  auto v_tile = [&](int idx) { load_tile(sV, vc + n * g.vs[0] + idx * g.vs[1] + hk * g.vs[3], g.vs[2], T); };
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[i][b] = 0.f;
  int idx = -1, k = next_slot(indices, zj, g, 0, idx), turn = 0;
  if (k < g.K) {
    load_tile(sQ, q + n * g.qs[0] + j * g.qs[1] + h * g.qs[2], g.qs[3], g.S);
    load_tile(sdO, dout + n * dos0 + j * dos1 + h * dos2, dos3, g.S);
    v_tile(idx);
    cp_commit();
    k_tile(idx);
    cp_commit();
  }
  while (k < g.K) {
    int idx_next = -1;
    const int k_next = next_slot(indices, zj, g, k + 1, idx_next);
    const long long slot = ((long long)zj * g.Hq + h) * g.K + k;
    const float w = weights[(long long)zj * g.K + k];
    float m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { const int r = own.row0 + 4 * i; m[i] = r < g.S ? lse[slot * g.S + r] : 0.f; }
    float s[4][8], dp[4][8];
    cp_wait<1>();                              // Q, dO and V are here
    unit_sync();
    mma_nt(sdO, sV, own, dp);
    cp_wait<0>();                              // K is here
    unit_sync();                           // and every warp is done with V
    if (k_next < g.K) v_tile(idx_next);
    cp_commit();
    mma_nt(sQ, sK, own, s);
    float di_sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = own.row0 + 4 * i;
      const bool live = r < g.S;
      float di = 0.f;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        s[i][b] = live ? exp2f(s[i][b] * c2 - m[i]) : 0.f;
        di = fmaf(s[i][b], dp[i][b], di);
      }
      di = row_sum(di);
      if (own.tx == 0) {
        di_sum += di;
        row_di[slot * T + r] = di;
      }
#pragma unroll
      for (int b = 0; b < 8; ++b) s[i][b] = s[i][b] * w * (dp[i][b] - di);
    }
    put_rows(sdS, own, s);
    // dw: the rows of a warp, then the warps, in a fixed order
#pragma unroll
    for (int of = 16; of >= 8; of >>= 1) di_sum += __shfl_xor_sync(0xffffffffu, di_sum, of);
    if ((threadIdx.x & 31) == 0) red[turn][threadIdx.x >> 5] = di_sum;
    __syncwarp();
    mma_nn_acc(sdS, sK, own, acc);
    unit_sync();                           // every warp is done with K
    if (PARTS == 1 && threadIdx.x == 0) dw_part[slot] = ((red[turn][0] + red[turn][1]) + red[turn][2]) + red[turn][3];
    if (PARTS == 4 && threadIdx.x < 4) dw_part[slot * 4 + threadIdx.x] = red[turn][threadIdx.x];
    if (k_next < g.K) k_tile(idx_next);
    cp_commit();
    k = k_next;
    idx = idx_next;
    turn ^= 1;
  }
  store_rows(dq + n * g.os[0] + j * g.os[1] + h * g.os[2], g.os[3], g.S, own, acc, g.sm_scale);
}

// ------------------------------------------------------------------------------------
// backward, kv-major: one (sequence n, cache chunk c, kv head).  Loops over every (query chunk j, slot k) that
// retrieved the chunk and over the q heads of the group, on transposed scores: rows = the chunk's keys.
// ------------------------------------------------------------------------------------
constexpr int BWD_KV_UNIT_SMEM = (4 * TILE + TILE_P) * sizeof(float);
template <typename E>
__device__ __forceinline__ void bwd_kv_unit(float* smem, const int4 unit, int hk, const E* __restrict__ q, const E* __restrict__ kc, const E* __restrict__ vc,
                                            const float* __restrict__ weights, const E* __restrict__ dout, const float* __restrict__ lse,
                                            const float* __restrict__ row_di, E* __restrict__ dk, E* __restrict__ dv, const Csr& csr, const Geom& g,
                                            long long dos0, long long dos1, long long dos2, long long dos3,
                                            long long dks0, long long dks1, long long dks2, long long dks3,
                                            long long dvs0, long long dvs1, long long dvs2, long long dvs3) {
  float *sK = smem, *sV = sK + TILE, *sQ = sV + TILE, *sdO = sQ + TILE, *sP = sdO + TILE;
  const int nc = unit.z;
  const int n = nc / g.C, c = nc % g.C;
  const Own own;
  const float c2 = g.sm_scale * GCA_LOG2E;
  float aK[4][8], aV[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < 8; ++b) { aK[i][b] = 0.f; aV[i][b] = 0.f; }
  // steps: (entry, q head of the group)
  const int steps = (unit.y - unit.x) * g.G;
  auto step_of = [&](int t, int& j, int& k, int& h) {
    const int e = t / g.G, entry = (int)(csr.sorted_keys[unit.x + e] & 0xffffffffull);
    j = entry / g.K;
    k = entry - j * g.K;
    h = hk * g.G + (t - e * g.G);
  };
  auto q_tile = [&](int j, int h) { load_tile(sQ, q + n * g.qs[0] + j * g.qs[1] + h * g.qs[2], g.qs[3], g.S); };
  auto o_tile = [&](int j, int h) { load_tile(sdO, dout + n * dos0 + j * dos1 + h * dos2, dos3, g.S); };
  int j = 0, k = 0, h = 0;
  if (steps > 0) {
    step_of(0, j, k, h);
    load_tile(sK, kc + n * g.ks[0] + c * g.ks[1] + hk * g.ks[3], g.ks[2], T);
    load_tile(sV, vc + n * g.vs[0] + c * g.vs[1] + hk * g.vs[3], g.vs[2], T);
    q_tile(j, h);
    o_tile(j, h);
    cp_commit();
  }
  for (int t = 0; t < steps; ++t) {
    const long long zj = (long long)n * g.J + j, slot = (zj * g.Hq + h) * g.K + k;
    const float w = weights[zj * g.K + k];
    float m[8], di[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int r = own.tx + 8 * b;
      m[b] = r < g.S ? lse[slot * g.S + r] : INFINITY;            // exp2(x - inf) = 0: rows past the end do not count
      di[b] = r < g.S ? row_di[slot * T + r] : 0.f;
    }
    if (t + 1 < steps) step_of(t + 1, j, k, h);
    cp_wait<0>();
    unit_sync();
    float p[4][8], dp[4][8];
    mma_nt(sK, sQ, own, p);
    mma_nt(sV, sdO, own, dp);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        p[i][b] = exp2f(p[i][b] * c2 - m[b]) * w;
        dp[i][b] = p[i][b] * (dp[i][b] - di[b]);
      }
    put_rows(sP, own, p);
    __syncwarp();
    mma_nn_acc(sP, sdO, own, aV);              // dV[key][d] += sum_row (w P)[row][key] dO[row][d]
    unit_sync();                           // every warp is done with dO
    if (t + 1 < steps) o_tile(j, h);
    put_rows(sP, own, dp);
    __syncwarp();
    mma_nn_acc(sP, sQ, own, aK);               // dK[key][d] += sum_row dS[row][key] Q[row][d]
    unit_sync();
    if (t + 1 < steps) q_tile(j, h);
    cp_commit();
  }
  store_rows(dk + n * dks0 + c * dks1 + hk * dks3, dks2, T, own, aK, g.sm_scale);
  store_rows(dv + n * dvs0 + c * dvs1 + hk * dvs3, dvs2, T, own, aV, 1.0f);
}

}  // namespace

}  // namespace gca
