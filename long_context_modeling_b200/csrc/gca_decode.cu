// GCA forward for a handful of query rows (autoregressive decode: 1 or 2 rows per
// sequence).  The work is a stream over K retrieved chunks x (K tile + V tile) per
// (sequence, kv head): HBM-bound, no tensor cores.  Two kernels: up to four rows per kv head (the
// model's decode step) take `decode_rows_kernel`, which streams the tiles through registers (see
// its comment); 5-16 rows take `decode_kernel`, described here.  Blocks are persistent (one per SM: each
// warp keeps a K and a V tile, 128 KB per block) and walk the (n, j, kv head) items; each warp
// owns whole slots and fetches its slot's two 8 KB tiles with two TMA copies (retrieved chunk
// index = tensor coordinate) onto two mbarriers of its own, so nothing is staged through
// registers.  As soon as a warp has scored its queries against the K tile it puts the K tile
// of its NEXT slot in flight -- of the next item when this one has no more slots for it -- and
// likewise the V tile after P.V: the loads of an item run under the arithmetic, the block-wide
// merge and the output store of the one before.  The K tile lands 128-byte-swizzled
// (conflict-free row reads), the V tile plain.  A warp scores the R = G*S query rows against
// the 64 keys (two keys per lane), normalises inside the warp and accumulates its weighted
// P.V in registers; the per-warp partial outputs are summed in warp order, so the result does
// not depend on scheduling.
#include "gca_common.cuh"
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

namespace gca {

namespace {

using namespace sm100;

constexpr int T = 64;
constexpr int NWARPS = 8;
constexpr int TILE_BYTES = T * T * 2;      // one bf16 tile

__device__ __forceinline__ float bf_lo(unsigned v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(unsigned v) { return __uint_as_float(v & 0xffff0000u); }

struct DecParams {
  CUtensorMap tm_k, tm_v;
  const __nv_bfloat16* q;
  const int32_t* indices;
  const float* weights;
  __nv_bfloat16* out;
  int32_t* status;
  Geom g;
};

template <int R>
__global__ void __launch_bounds__(NWARPS * 32)
decode_kernel(const __grid_constant__ DecParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* tile_k = smem + warp * 2 * TILE_BYTES;                                       // swizzled
  uint8_t* tile_v = tile_k + TILE_BYTES;                                                // plain
  float* sQ_all = reinterpret_cast<float*>(smem + NWARPS * 2 * TILE_BYTES);             // [2][R x 64] scaled queries
  float* part_all = sQ_all + 2 * R * T;                                                 // [2][NWARPS][R x 64] partial outputs
  uint64_t* bars = reinterpret_cast<uint64_t*>(part_all + 2 * NWARPS * R * T);          // [NWARPS][K, V]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * NWARPS);
  const Geom& g = p.g;
  const int items = g.N * g.J * g.Hkv;
  const int rows = g.G * g.S;                                    // <= R
  const float c2 = g.sm_scale * GCA_LOG2E;
  uint64_t* bar_k = &bars[2 * warp];
  uint64_t* bar_v = &bars[2 * warp + 1];

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * NWARPS; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  // This warp's slots, in order: (item, k) with k = warp, warp + 8, ... < K, then the next item.
  // `cur` is the slot whose tiles are (or are about to be) in the buffers; idx < 0: no copy.
  struct Slot { int item, k, idx; };
  auto load_idx = [&](int item, int k) -> int {
    const int zj = item / g.Hkv;
    const int v = slot_chunk(p.indices, zj, g.K, k);
    if (v >= g.C) { if (p.status && lane == 0) atomicOr(p.status, GCA_STATUS_BAD_INDEX); return -1; }
    return v;
  };
  auto next_slot = [&](const Slot& s) -> Slot {
    Slot t;
    t.item = s.item; t.k = s.k + NWARPS;
    if (t.k >= g.K) { t.item = s.item + (int)gridDim.x; t.k = warp; }
    t.idx = (t.item < items && t.k < g.K) ? load_idx(t.item, t.k) : -1;
    return t;
  };
  auto issue = [&](const Slot& s, bool is_v) {
    if (lane == 0) {
      const int zj = s.item / g.Hkv, hk = s.item - zj * g.Hkv;
      uint64_t* bar = is_v ? bar_v : bar_k;
      mbar_arrive_expect_tx(bar, TILE_BYTES);
      tma_load_5d(is_v ? tile_v : tile_k, is_v ? &p.tm_v : &p.tm_k, bar, 0, 0, hk, s.idx, zj / g.J);
    }
  };

  Slot cur;
  cur.item = blockIdx.x; cur.k = warp;
  cur.idx = (cur.item < items && cur.k < g.K) ? load_idx(cur.item, cur.k) : -1;
  bool in_k = false, in_v = false;               // a copy is in flight (or landed, unread) in the K / V buffer
  if (cur.idx >= 0) { issue(cur, false); issue(cur, true); in_k = in_v = true; }
  uint32_t ph_k = 0, ph_v = 0;
  bool ok = true;

  int par = 0;
  for (int item = blockIdx.x; item < items; item += gridDim.x, par ^= 1) {
    const int zj = item / g.Hkv, hk = item - zj * g.Hkv;
    const int n = zj / g.J, j = zj - n * g.J;
    float* sQ = sQ_all + par * R * T;
    float* part = part_all + par * NWARPS * R * T;
    for (int i = threadIdx.x; i < R * T; i += NWARPS * 32) {
      const int r = i >> 6, d = i & 63;
      float v = 0.f;
      if (r < rows) {
        const int gi = r / g.S, s = r % g.S;
        v = __bfloat162float(p.q[n * g.qs[0] + j * g.qs[1] + (hk * g.G + gi) * g.qs[2] + s * g.qs[3] + d]);
      }
      sQ[i] = v * c2;
    }
    __syncthreads();

    float o[R][2];
#pragma unroll
    for (int r = 0; r < R; ++r) { o[r][0] = 0.f; o[r][1] = 0.f; }

    while (cur.item == item && cur.k < g.K) {
      const Slot nxt = next_slot(cur);           // its index load overlaps the waits below
      float pr[R][2];
      if (cur.idx >= 0 && ok) {
        const float w = p.weights[(long long)zj * g.K + cur.k];
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar_k, ph_k, abort_flag));
        ph_k ^= 1;
        in_k = false;
        if (ok) {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            pr[r][0] = pr[r][1] = 0.f;
            if (r >= rows) continue;
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int pc = 0; pc < 8; ++pc) {
              const uint4 a = *reinterpret_cast<const uint4*>(tile_k + lane * 128 + ((pc ^ (lane & 7)) << 4));
              const uint4 b = *reinterpret_cast<const uint4*>(tile_k + (lane + 32) * 128 + ((pc ^ (lane & 7)) << 4));
              const float* qr = sQ + r * T + pc * 8;
              s0 = fmaf(qr[0], bf_lo(a.x), s0); s0 = fmaf(qr[1], bf_hi(a.x), s0);
              s0 = fmaf(qr[2], bf_lo(a.y), s0); s0 = fmaf(qr[3], bf_hi(a.y), s0);
              s0 = fmaf(qr[4], bf_lo(a.z), s0); s0 = fmaf(qr[5], bf_hi(a.z), s0);
              s0 = fmaf(qr[6], bf_lo(a.w), s0); s0 = fmaf(qr[7], bf_hi(a.w), s0);
              s1 = fmaf(qr[0], bf_lo(b.x), s1); s1 = fmaf(qr[1], bf_hi(b.x), s1);
              s1 = fmaf(qr[2], bf_lo(b.y), s1); s1 = fmaf(qr[3], bf_hi(b.y), s1);
              s1 = fmaf(qr[4], bf_lo(b.z), s1); s1 = fmaf(qr[5], bf_hi(b.z), s1);
              s1 = fmaf(qr[6], bf_lo(b.w), s1); s1 = fmaf(qr[7], bf_hi(b.w), s1);
            }
            float m = fmaxf(s0, s1);
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, of));
            if (g.off_by_one > 0.f) m = fmaxf(m, 0.f);
            float p0 = exp2f(s0 - m), p1 = exp2f(s1 - m);
            float l = p0 + p1;
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) l += __shfl_xor_sync(0xffffffffu, l, of);
            if (g.off_by_one > 0.f) l += g.off_by_one * exp2f(-m);
            const float f = w / l;
            pr[r][0] = p0 * f; pr[r][1] = p1 * f;
          }
        }
      }
      // the K buffer has been read: the next slot's K tile goes in flight under the P.V below
      __syncwarp();
      if (nxt.idx >= 0 && ok) { issue(nxt, false); in_k = true; }
      if (cur.idx >= 0 && ok) {
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar_v, ph_v, abort_flag));
        ph_v ^= 1;
        in_v = false;
        if (ok) {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (r >= rows) break;
            float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
            for (int key = 0; key < 32; ++key) {
              const float pa = __shfl_sync(0xffffffffu, pr[r][0], key);
              const float pb = __shfl_sync(0xffffffffu, pr[r][1], key);
              const unsigned va = *reinterpret_cast<const unsigned*>(tile_v + key * 128 + lane * 4);
              const unsigned vb = *reinterpret_cast<const unsigned*>(tile_v + (key + 32) * 128 + lane * 4);
              a0 = fmaf(pa, bf_lo(va), a0); a1 = fmaf(pa, bf_hi(va), a1);
              a0 = fmaf(pb, bf_lo(vb), a0); a1 = fmaf(pb, bf_hi(vb), a1);
            }
            o[r][0] += a0; o[r][1] += a1;
          }
        }
      }
      __syncwarp();
      if (nxt.idx >= 0 && ok) { issue(nxt, true); in_v = true; }
      cur = nxt;
    }
    // cross-warp sum in warp order
#pragma unroll
    for (int r = 0; r < R; ++r) {
      part[(warp * R + r) * T + 2 * lane] = o[r][0];
      part[(warp * R + r) * T + 2 * lane + 1] = o[r][1];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < rows * T; i += NWARPS * 32) {
      const int r = i >> 6, d = i & 63;
      float t = 0.f;
#pragma unroll
      for (int wv = 0; wv < NWARPS; ++wv) t += part[(wv * R + r) * T + d];
      const int gi = r / g.S, s = r % g.S;
      p.out[n * g.os[0] + j * g.os[1] + (hk * g.G + gi) * g.os[2] + s * g.os[3] + d] = __float2bfloat16_rn(t);
    }
  }
  // a warp that gave up may still have copies in flight: wait for them (bounded) so nothing
  // lands in shared memory after the block has exited
  if (lane == 0) {
    if (in_k) for (int i = 0; i < (1 << 20); ++i) if (mbar_try_wait(bar_k, ph_k)) break;
    if (in_v) for (int i = 0; i < (1 << 20); ++i) if (mbar_try_wait(bar_v, ph_v)) break;
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicOr(p.status, GCA_STATUS_TIMEOUT);
}

// ---------------------------------------------------------------------------------------------
// Up to four query rows per kv head (the model's decode step: one row): no shared-memory staging at
// all.  One CTA per (sequence, query chunk, kv head), one warp per retrieved slot (slots k = warp,
// warp + 8, ...).  A warp load covers FOUR key rows of the slot's tile (8 lanes x 16 bytes per
// 128-byte row); every 8-lane group owns a stream of 16 keys with its own online-softmax state, the
// loads run four steps ahead of the arithmetic in registers, and nothing is waited for except the
// data itself.  Registers are capped so that three CTAs share an SM: 32 sequences x
// 12 heads = 384 CTAs run as one wave, where the persistent TMA kernel below needs a ragged third
// round of its 148 CTAs.  The four streams of a warp, then the slots in slot order, are merged in a
// fixed order: the result does not depend on scheduling.
struct RowState { float m, l, acc[8]; };
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void merge_state(RowState& a, float m2, float l2, const float* acc2) {
  const float m = fmaxf(a.m, m2);
  const float ca = (a.m == -INFINITY) ? 0.f : ex2f(a.m - m), cb = (m2 == -INFINITY) ? 0.f : ex2f(m2 - m);
  a.l = a.l * ca + l2 * cb;
#pragma unroll
  for (int i = 0; i < 8; ++i) a.acc[i] = a.acc[i] * ca + acc2[i] * cb;
  a.m = m;
}

template <int R>
__global__ void __launch_bounds__(NWARPS * 32, R == 1 ? 3 : (R == 2 ? 2 : 1))
decode_rows_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kc, const __nv_bfloat16* __restrict__ vc,
                   const int32_t* __restrict__ indices, const float* __restrict__ weights, __nv_bfloat16* __restrict__ out,
                   int32_t* status, const Geom g) {
  __shared__ float part[NWARPS][R][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, sub = lane & 7;
  const int item = blockIdx.x;
  const int zj = item / g.Hkv, hk = item - zj * g.Hkv;
  const int n = zj / g.J, j = zj - n * g.J;
  const int rows = g.G * g.S;                                    // <= R
  const float c2 = g.sm_scale * GCA_LOG2E;
  pdl_trigger();
  // While the kernel before is finishing, this warp's first K tile on its way into L2 (V as well, which fills the queues the
  // loads behind the wait need: no gain left).  The index may not be final yet, so it is a hint here, read past L1 and read
  // again below.
  if (warp < g.K) {
    int hint = warp;
    if (indices) asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(hint) : "l"(indices + (long long)zj * g.K + warp) : "memory");
    if (hint >= 0 && hint < g.C) {
      const __nv_bfloat16* kt = kc + n * g.ks[0] + hint * g.ks[1] + hk * g.ks[3] + lane * g.ks[2];
      asm volatile("prefetch.global.L2 [%0];" ::"l"(kt));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(kt + 32 * g.ks[2]));
    }
  }
  pdl_wait();
  float qv[R][8];
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int e = 0; e < 8; ++e) qv[r][e] = 0.f;
    if (r < rows) {
      const int gi = r / g.S, s = r - gi * g.S;
      const uint4 t = *reinterpret_cast<const uint4*>(q + n * g.qs[0] + j * g.qs[1] + (hk * g.G + gi) * g.qs[2] + s * g.qs[3] + sub * 8);
      const unsigned w4[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) { qv[r][2 * e] = bf_lo(w4[e]) * c2; qv[r][2 * e + 1] = bf_hi(w4[e]) * c2; }
    }
  }
  float o[R][8];                                 // this warp's weighted outputs, 8 columns per lane
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int e = 0; e < 8; ++e) o[r][e] = 0.f;
  for (int k = warp; k < g.K; k += NWARPS) {
    const int idx = slot_chunk(indices, zj, g.K, k);
    if (idx < 0) continue;                                       // padding slot (warp-uniform)
    if (idx >= g.C) { if (status && lane == 0) atomicOr(status, GCA_STATUS_BAD_INDEX); continue; }
    const float w = weights[(long long)zj * g.K + k];
    const __nv_bfloat16* kb = kc + n * g.ks[0] + idx * g.ks[1] + hk * g.ks[3] + sub * 8 + grp * g.ks[2];
    const __nv_bfloat16* vb = vc + n * g.vs[0] + idx * g.vs[1] + hk * g.vs[3] + sub * 8 + grp * g.vs[2];
    RowState st[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      st[r].m = -INFINITY; st[r].l = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) st[r].acc[e] = 0.f;
    }
    // 16 steps of 4 keys, four steps at a time: the next four steps' rows are requested as soon as the registers are read, and
    // the four steps share one maximum and one rescaling (a step of its own each was a chain of ~200 cycles)
    uint4 kq[4], vq[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      kq[s] = *reinterpret_cast<const uint4*>(kb); kb += 4 * g.ks[2];
      vq[s] = *reinterpret_cast<const uint4*>(vb); vb += 4 * g.vs[2];
    }
#pragma unroll 1
    for (int b4 = 0; b4 < 16; b4 += 4) {
      float sc[R][4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const unsigned kw[4] = {kq[s].x, kq[s].y, kq[s].z, kq[s].w};
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float t = 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) { t = fmaf(qv[r][2 * e], bf_lo(kw[e]), t); t = fmaf(qv[r][2 * e + 1], bf_hi(kw[e]), t); }
          sc[r][s] = t;
        }
        if (b4 + 4 < 16) { kq[s] = *reinterpret_cast<const uint4*>(kb); kb += 4 * g.ks[2]; }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int of = 1; of < 8; of <<= 1)
#pragma unroll
          for (int s = 0; s < 4; ++s) sc[r][s] += __shfl_xor_sync(0xffffffffu, sc[r][s], of);
        const float m = fmaxf(st[r].m, fmaxf(fmaxf(sc[r][0], sc[r][1]), fmaxf(sc[r][2], sc[r][3])));
        const float corr = ex2f(st[r].m - m);
        st[r].m = m;
#pragma unroll
        for (int s = 0; s < 4; ++s) sc[r][s] = ex2f(sc[r][s] - m);
        st[r].l = st[r].l * corr + ((sc[r][0] + sc[r][1]) + (sc[r][2] + sc[r][3]));
#pragma unroll
        for (int e = 0; e < 8; ++e) st[r].acc[e] *= corr;
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const unsigned vw[4] = {vq[s].x, vq[s].y, vq[s].z, vq[s].w};
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            st[r].acc[2 * e] = fmaf(sc[r][s], bf_lo(vw[e]), st[r].acc[2 * e]);
            st[r].acc[2 * e + 1] = fmaf(sc[r][s], bf_hi(vw[e]), st[r].acc[2 * e + 1]);
          }
        if (b4 + 4 < 16) { vq[s] = *reinterpret_cast<const uint4*>(vb); vb += 4 * g.vs[2]; }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int of = 8; of <= 16; of <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, st[r].m, of), l2 = __shfl_xor_sync(0xffffffffu, st[r].l, of);
        float a2[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) a2[e] = __shfl_xor_sync(0xffffffffu, st[r].acc[e], of);
        merge_state(st[r], m2, l2, a2);
      }
      // softmax over this slot's 64 keys (optionally with the off-by-one term), weighted by w
      float mm = st[r].m, ll = st[r].l;
      if (g.off_by_one > 0.f) {
        const float m1 = fmaxf(mm, 0.f);
        ll = ll * ex2f(mm - m1) + g.off_by_one * ex2f(-m1);
        const float sc1 = ex2f(mm - m1);
#pragma unroll
        for (int e = 0; e < 8; ++e) st[r].acc[e] *= sc1;
      }
      const float f = w / ll;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[r][e] = fmaf(st[r].acc[e], f, o[r][e]);
    }
  }
  if (grp == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int e = 0; e < 8; ++e) part[warp][r][sub * 8 + e] = o[r][e];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rows * 64; i += NWARPS * 32) {
    const int r = i >> 6, d = i & 63;
    float t = 0.f;
#pragma unroll
    for (int wv = 0; wv < NWARPS; ++wv) t += part[wv][r][d];
    const int gi = r / g.S, s = r - gi * g.S;
    out[n * g.os[0] + j * g.os[1] + (hk * g.G + gi) * g.os[2] + s * g.os[3] + d] = __float2bfloat16_rn(t);
  }
}

// The same for so few (sequence, kv head) items that the SMs are not all busy: WPS warps share a slot (64 / WPS keys each, all
// their loads in flight at once), the partial softmax states meet in shared memory.  One sequence, 12 heads, K = 8, behind the
// projection it depends on: 6.0 -> ~4 us.
template <int R, int WPS>
__global__ void __launch_bounds__(NWARPS * WPS * 32)
decode_split_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kc, const __nv_bfloat16* __restrict__ vc,
                    const int32_t* __restrict__ indices, const float* __restrict__ weights, __nv_bfloat16* __restrict__ out,
                    int32_t* status, const Geom g) {
  constexpr int STEPS = 16 / WPS, PITCH = 66;                    // (maximum, sum, 64 outputs)
  extern __shared__ float part[];                                // [K][WPS][R][PITCH]
  __shared__ float slot_w[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, sub = lane & 7;
  const int item = blockIdx.x;
  const int zj = item / g.Hkv, hk = item - zj * g.Hkv;
  const int n = zj / g.J, j = zj - n * g.J;
  const int rows = g.G * g.S;
  const float c2 = g.sm_scale * GCA_LOG2E;
  pdl_trigger();
  pdl_wait();
  uint4 qv[R];                                                   // this lane's 8 query values of every row, as they came
#pragma unroll
  for (int r = 0; r < R; ++r) {
    qv[r] = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      const int gi = r / g.S, s = r - gi * g.S;
      qv[r] = *reinterpret_cast<const uint4*>(q + n * g.qs[0] + j * g.qs[1] + (hk * g.G + gi) * g.qs[2] + s * g.qs[3] + sub * 8);
    }
  }
  const int share = warp % WPS;
  for (int k = warp / WPS; k < g.K; k += NWARPS) {
    const int idx = slot_chunk(indices, zj, g.K, k);
    const bool live = idx >= 0 && idx < g.C;
    if (share == 0 && lane == 0) {
      if (idx >= g.C && status) atomicOr(status, GCA_STATUS_BAD_INDEX);
      slot_w[k] = live ? weights[(long long)zj * g.K + k] : 0.f;
    }
    if (!live) continue;
    const int key0 = share * (64 / WPS) + grp;
    const __nv_bfloat16* kb = kc + n * g.ks[0] + idx * g.ks[1] + hk * g.ks[3] + sub * 8;
    const __nv_bfloat16* vb = vc + n * g.vs[0] + idx * g.vs[1] + hk * g.vs[3] + sub * 8;
    uint4 kq[STEPS], vq[STEPS];
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      kq[s] = *reinterpret_cast<const uint4*>(kb + (key0 + s * 4) * g.ks[2]);
      vq[s] = *reinterpret_cast<const uint4*>(vb + (key0 + s * 4) * g.vs[2]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float sc[STEPS], m = -INFINITY;
      const unsigned qw[4] = {qv[r].x, qv[r].y, qv[r].z, qv[r].w};
#pragma unroll
      for (int s = 0; s < STEPS; ++s) {
        const unsigned kw[4] = {kq[s].x, kq[s].y, kq[s].z, kq[s].w};
        float t = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) { t = fmaf(bf_lo(qw[e]), bf_lo(kw[e]), t); t = fmaf(bf_hi(qw[e]), bf_hi(kw[e]), t); }
        sc[s] = t * c2;
      }
#pragma unroll
      for (int of = 1; of < 8; of <<= 1)
#pragma unroll
        for (int s = 0; s < STEPS; ++s) sc[s] += __shfl_xor_sync(0xffffffffu, sc[s], of);
#pragma unroll
      for (int s = 0; s < STEPS; ++s) m = fmaxf(m, sc[s]);
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
      float l = 0.f, acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll
      for (int s = 0; s < STEPS; ++s) {
        const float pr = ex2f(sc[s] - m);
        l += pr;
        const unsigned vw[4] = {vq[s].x, vq[s].y, vq[s].z, vq[s].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) { acc[2 * e] = fmaf(pr, bf_lo(vw[e]), acc[2 * e]); acc[2 * e + 1] = fmaf(pr, bf_hi(vw[e]), acc[2 * e + 1]); }
      }
#pragma unroll
      for (int of = 8; of <= 16; of <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, of);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], of);
      }
      float* dst = part + ((k * WPS + share) * R + r) * PITCH;
      if (lane == 0) { dst[0] = m; dst[1] = l; }
      if (grp == 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[2 + sub * 8 + e] = acc[e];
      }
    }
  }
  __syncthreads();
  // out = sum over slots of w * (merged numerator) / (merged sum), in slot order
  for (int i = threadIdx.x; i < rows * 64; i += NWARPS * WPS * 32) {
    const int r = i >> 6, d = i & 63;
    float t = 0.f;
    for (int k = 0; k < g.K; ++k) {
      const float w = slot_w[k];
      const int idx = slot_chunk(indices, zj, g.K, k);
      if (idx < 0 || idx >= g.C) continue;
      const float* src = part + (k * WPS * R + r) * PITCH;
      float m = g.off_by_one > 0.f ? 0.f : -INFINITY;
#pragma unroll
      for (int x = 0; x < WPS; ++x) m = fmaxf(m, src[x * R * PITCH]);
      float l = g.off_by_one > 0.f ? g.off_by_one * ex2f(-m) : 0.f, o = 0.f;
#pragma unroll
      for (int x = 0; x < WPS; ++x) {
        const float c = ex2f(src[x * R * PITCH] - m);
        l = fmaf(src[x * R * PITCH + 1], c, l);
        o = fmaf(src[x * R * PITCH + 2 + d], c, o);
      }
      t = fmaf(o, w / l, t);
    }
    const int gi = r / g.S, s = r - gi * g.S;
    out[n * g.os[0] + j * g.os[1] + (hk * g.G + gi) * g.os[2] + s * g.os[3] + d] = __float2bfloat16_rn(t);
  }
}

template <int R>
int launch_decode_r(const DecParams& p, int blocks, int sms, cudaStream_t stream) {
  const size_t smem = NWARPS * 2 * TILE_BYTES + 2 * (1 + NWARPS) * R * T * sizeof(float) + 256 + 1024;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(decode_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  decode_kernel<R><<<(unsigned)(blocks < sms ? blocks : sms), NWARPS * 32, smem, stream>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace

// bf16, G*S <= 16 rows.  Returns GCA_ERR_ALGO when the problem is outside that envelope.
int launch_decode(const GcaFwdArgs& a, int sms, cudaStream_t stream) {
  if (a.dtype != GCA_BF16) return GCA_ERR_ALGO;
  DecParams p;
  p.q = (const __nv_bfloat16*)a.q; p.indices = a.indices; p.weights = a.weights;
  p.out = (__nv_bfloat16*)a.out; p.status = a.status;
  Geom& g = p.g;
  g.N = a.N; g.J = a.J; g.Hq = a.Hq; g.Hkv = a.Hkv; g.S = a.S; g.L = a.L; g.D = a.D; g.K = a.K; g.C = a.C;
  g.G = a.Hq / a.Hkv;
  for (int i = 0; i < 4; ++i) { g.qs[i] = a.q_stride[i]; g.os[i] = a.o_stride[i]; g.ks[i] = a.k_stride[i]; g.vs[i] = a.v_stride[i]; }
  g.sm_scale = a.sm_scale; g.off_by_one = a.off_by_one;
  const int rows = g.G * a.S;
  const int blocks = a.N * a.J * a.Hkv;
  // up to four rows: the register-streaming kernel (needs 16-byte aligned 128-byte head rows, which
  // the argument checks of the entry point guarantee for q and the caches)
  bool vec16 = true;                  // every 64-element head row of q and the caches starts on a 16-byte boundary
  for (int i = 0; i < 4; ++i) vec16 = vec16 && a.q_stride[i] % 8 == 0 && a.k_stride[i] % 8 == 0 && a.v_stride[i] % 8 == 0;
  vec16 = vec16 && ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k_cache) | reinterpret_cast<uintptr_t>(a.v_cache)) & 15u) == 0;
  if (rows <= 4 && blocks > 0 && a.D == 64 && a.L == 64 && vec16) {
    auto q = (const __nv_bfloat16*)a.q; auto kc = (const __nv_bfloat16*)a.k_cache; auto vc = (const __nv_bfloat16*)a.v_cache;
    auto out = (__nv_bfloat16*)a.out;
    // warps per slot while whole SMs would be idle (the states of all slots fit 48 KB of shared memory)
    const int wps = rows <= 2 && blocks <= sms ? 4 : rows <= 2 && blocks <= 2 * sms ? 2 : 1;
    const size_t smem = (size_t)a.K * wps * (rows <= 1 ? 1 : 2) * 66 * sizeof(float);
    auto run = [&](auto kernel, int threads, size_t bytes) {
      return (int)launch_dependent(kernel, dim3((unsigned)blocks), dim3(threads), bytes, stream, q, kc, vc, a.indices, a.weights, out, a.status, g);
    };
    if (wps > 1 && smem <= 48 * 1024) {
      if (rows <= 1) return wps == 4 ? run(decode_split_kernel<1, 4>, NWARPS * 128, smem) : run(decode_split_kernel<1, 2>, NWARPS * 64, smem);
      return wps == 4 ? run(decode_split_kernel<2, 4>, NWARPS * 128, smem) : run(decode_split_kernel<2, 2>, NWARPS * 64, smem);
    }
    if (rows <= 1) return run(decode_rows_kernel<1>, NWARPS * 32, 0);
    if (rows <= 2) return run(decode_rows_kernel<2>, NWARPS * 32, 0);
    return run(decode_rows_kernel<4>, NWARPS * 32, 0);
  }
  int rc;
  if ((rc = make_tile_map_5d(&p.tm_k, a.k_cache, 64, 64, a.Hkv, a.C, a.N, a.k_stride[2], a.k_stride[3], a.k_stride[1], a.k_stride[0], 1, true))) return rc;
  if ((rc = make_tile_map_5d(&p.tm_v, a.v_cache, 64, 64, a.Hkv, a.C, a.N, a.v_stride[2], a.v_stride[3], a.v_stride[1], a.v_stride[0], 1, false))) return rc;
  if (rows <= 8) return launch_decode_r<8>(p, blocks, sms, stream);
  if (rows <= 16) return launch_decode_r<16>(p, blocks, sms, stream);
  return GCA_ERR_ALGO;
}

}  // namespace gca
