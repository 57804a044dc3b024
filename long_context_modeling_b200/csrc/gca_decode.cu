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
// Up to four query rows per kv head (the model's decode step: one row): no shared-memory staging at all.  WPS warps per
// retrieved slot (64 / WPS keys each), the slots of an item dealt out over the warps of a CTA or of a cluster of them.  A warp
// load covers FOUR key rows of the slot's tile (8 lanes x 16 bytes per 128-byte row); every 8-lane group owns a stream of keys
// with its own online-softmax state, the loads run four steps ahead of the arithmetic in registers, and nothing is waited for
// except the data itself.  The streams of a warp, the warps of a slot, the slots and the CTAs of a cluster are merged in a fixed
// order: the result does not depend on scheduling.
// Bound: HBM for many items (32 sequences x 12 heads x 8 slots: 11.0 us, 7.7 at the copy rate; at most eight warps an item and a
// step of its own for every four keys took 11.6), else latency: launch, one round of loads, the merges (one row, 132 items, K = 13:
// 7.4 us against 8.7; two rows, 8 items, K = 16: 4.2 against 18.1, 96 items, K = 15: 7.8 against 17.9).  What each split gains is
// said at decode_plan().
struct RowState { float m, l; float2 acc[4]; };
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 bf2(unsigned v) { return make_float2(bf_lo(v), bf_hi(v)); }
__device__ __forceinline__ float2 splat(float x) { return make_float2(x, x); }
// Registers a thread and the most warps a CTA of decode_rows_kernel<rows, wps> has.
template <int R, int WPS> constexpr int ROW_REGS = R > 1 ? 128 : WPS == 4 ? 64 : 80;
template <int R, int WPS> constexpr int ROW_WARPS = R > 1 ? 16 : WPS == 4 ? 32 : 24;
constexpr int STATE = 66;                                        // maximum, sum, 64 outputs

template <int R, int WPS>
__global__ void __maxnreg__((ROW_REGS<R, WPS>))
decode_rows_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kc, const __nv_bfloat16* __restrict__ vc,
                   const int32_t* __restrict__ indices, const float* __restrict__ weights, __nv_bfloat16* __restrict__ out,
                   int32_t* status, const Geom g, int ctas) {
  constexpr int BATCHES = 4 / WPS;                               // of four steps of four keys
  constexpr int WARPS = ROW_WARPS<R, WPS>;
  __shared__ float part[WARPS][R][WPS > 1 ? STATE : 64];        // a warp's weighted outputs over its slots; WPS > 1: its part of its slot's state
  __shared__ float total[R][64];                                 // this CTA's sum
  __shared__ float slot_w[WARPS];
  __shared__ bool slot_reads[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, sub = lane & 7;
  const int warps = blockDim.x >> 5, slots = warps / WPS;        // of the CTA
  const int unit = blockIdx.x / ctas, rank = blockIdx.x - unit * ctas;
  const bool pairs = R > 1 && g.G * g.S > R;                     // three or four rows: an item's two pairs follow one another
  const int item = pairs ? unit >> 1 : unit, row0 = pairs ? (unit & 1) * R : 0, rows = min(R, g.G * g.S - row0);      // this CTA's rows of the kv head
  const int zj = item / g.Hkv, hk = item - zj * g.Hkv;
  const int n = zj / g.J, j = zj - n * g.J;
  const float c2 = g.sm_scale * GCA_LOG2E;
  const int k0 = rank * slots + warp / WPS, share = warp % WPS;
  pdl_trigger();
  // While the kernel before is finishing, this warp's first K tile on its way into L2 (V as well, which fills the queues the
  // loads behind the wait need: no gain left).  The index may not be final yet, so it is a hint here, read past L1 and read
  // again below.
  if (k0 < g.K) {
    int hint = k0;
    if (indices) asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(hint) : "l"(indices + (long long)zj * g.K + k0) : "memory");
    if (hint >= 0 && hint < g.C) {
      const __nv_bfloat16* kt = kc + n * g.ks[0] + hint * g.ks[1] + hk * g.ks[3] + (share * (64 / WPS) + lane % (64 / WPS)) * g.ks[2];
      asm volatile("prefetch.global.L2 [%0];" ::"l"(kt));
      if (WPS == 1) asm volatile("prefetch.global.L2 [%0];" ::"l"(kt + 32 * g.ks[2]));
    }
  }
  pdl_wait();
  uint4 qv[R];                                                   // this lane's 8 query values of every row, as they came
#pragma unroll
  for (int r = 0; r < R; ++r) {
    qv[r] = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      const int gi = (row0 + r) / g.S, s = row0 + r - gi * g.S;
      qv[r] = *reinterpret_cast<const uint4*>(q + n * g.qs[0] + j * g.qs[1] + (hk * g.G + gi) * g.qs[2] + s * g.qs[3] + sub * 8);
    }
  }
  if (WPS == 1) {
    for (int i = lane; i < R * 64; i += 32) (&part[warp][0][0])[i] = 0.f;
    __syncwarp();
  } else if (share == 0 && lane == 0) slot_reads[warp / WPS] = false;
  for (int k = k0; k < g.K; k += ctas * slots) {
    const int idx = slot_chunk(indices, zj, g.K, k);
    if (idx < 0) continue;                                       // padding slot (warp-uniform)
    if (idx >= g.C) { if (status && share == 0 && lane == 0) atomicOr(status, GCA_STATUS_BAD_INDEX); continue; }
    const float w = weights[(long long)zj * g.K + k];
    const int key0 = share * (64 / WPS) + grp;
    const __nv_bfloat16* kb = kc + n * g.ks[0] + idx * g.ks[1] + hk * g.ks[3] + sub * 8 + key0 * g.ks[2];
    const __nv_bfloat16* vb = vc + n * g.vs[0] + idx * g.vs[1] + hk * g.vs[3] + sub * 8 + key0 * g.vs[2];
    RowState st[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      st[r].m = -INFINITY; st[r].l = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) st[r].acc[e] = splat(0.f);
    }
    // steps of 4 keys, four steps at a time: the next four steps' rows are requested as soon as the registers are read, and
    // the four steps share one maximum and one rescaling (a step of its own each was a chain of ~200 cycles)
    uint4 kq[4], vq[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      kq[s] = *reinterpret_cast<const uint4*>(kb); kb += 4 * g.ks[2];
      vq[s] = *reinterpret_cast<const uint4*>(vb); vb += 4 * g.vs[2];
    }
#pragma unroll 1
    for (int b = 0; b < BATCHES; ++b) {
      float sc[R][4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const float2 k2[4] = {bf2(kq[s].x), bf2(kq[s].y), bf2(kq[s].z), bf2(kq[s].w)};
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float2 t = __fmul2_rn(bf2(qv[r].x), k2[0]);
          t = __ffma2_rn(bf2(qv[r].y), k2[1], t);
          t = __ffma2_rn(bf2(qv[r].z), k2[2], t);
          t = __ffma2_rn(bf2(qv[r].w), k2[3], t);
          sc[r][s] = t.x + t.y;
        }
        if (b + 1 < BATCHES) { kq[s] = *reinterpret_cast<const uint4*>(kb); kb += 4 * g.ks[2]; }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int of = 1; of < 8; of <<= 1)
#pragma unroll
          for (int s = 0; s < 4; ++s) sc[r][s] += __shfl_xor_sync(0xffffffffu, sc[r][s], of);
        const float m = fmaxf(st[r].m, fmaxf(fmaxf(sc[r][0], sc[r][1]), fmaxf(sc[r][2], sc[r][3])) * c2);
        const float corr = ex2f(st[r].m - m);
        st[r].m = m;
#pragma unroll
        for (int s = 0; s < 4; ++s) sc[r][s] = ex2f(fmaf(sc[r][s], c2, -m));
        st[r].l = fmaf(st[r].l, corr, (sc[r][0] + sc[r][1]) + (sc[r][2] + sc[r][3]));
        if (BATCHES > 1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) st[r].acc[e] = __fmul2_rn(st[r].acc[e], splat(corr));
        }
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const float2 v2[4] = {bf2(vq[s].x), bf2(vq[s].y), bf2(vq[s].z), bf2(vq[s].w)};
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) st[r].acc[e] = __ffma2_rn(splat(sc[r][s]), v2[e], st[r].acc[e]);
        if (b + 1 < BATCHES) { vq[s] = *reinterpret_cast<const uint4*>(vb); vb += 4 * g.vs[2]; }
      }
    }
    if (WPS > 1 && share == 0 && lane == 0) { slot_w[warp / WPS] = w; slot_reads[warp / WPS] = true; }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      // the four streams: one maximum, then plain sums
      float m = fmaxf(st[r].m, __shfl_xor_sync(0xffffffffu, st[r].m, 8));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
      const float corr = ex2f(st[r].m - m);
      float l = st[r].l * corr;
#pragma unroll
      for (int e = 0; e < 4; ++e) st[r].acc[e] = __fmul2_rn(st[r].acc[e], splat(corr));
#pragma unroll
      for (int of = 8; of <= 16; of <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, of);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          st[r].acc[e].x += __shfl_xor_sync(0xffffffffu, st[r].acc[e].x, of);
          st[r].acc[e].y += __shfl_xor_sync(0xffffffffu, st[r].acc[e].y, of);
        }
      }
      if (WPS > 1) {
        float* dst = part[warp][r];
        if (lane == 0) { dst[0] = m; dst[1] = l; }
        if (grp == 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e) { dst[2 + sub * 8 + 2 * e] = st[r].acc[e].x; dst[2 + sub * 8 + 2 * e + 1] = st[r].acc[e].y; }
        }
      } else {
        // softmax over this slot's 64 keys (optionally with the off-by-one term), weighted by w
        float f = 1.f;
        if (g.off_by_one > 0.f) {
          const float m1 = fmaxf(m, 0.f);
          f = ex2f(m - m1);
          l = l * f + g.off_by_one * ex2f(-m1);
        }
        f *= w / l;
        if (grp == 0) {
          float4* dst = reinterpret_cast<float4*>(&part[warp][r][sub * 8]);
          const float4 a = dst[0], b = dst[1];
          dst[0] = make_float4(fmaf(st[r].acc[0].x, f, a.x), fmaf(st[r].acc[0].y, f, a.y), fmaf(st[r].acc[1].x, f, a.z), fmaf(st[r].acc[1].y, f, a.w));
          dst[1] = make_float4(fmaf(st[r].acc[2].x, f, b.x), fmaf(st[r].acc[2].y, f, b.y), fmaf(st[r].acc[3].x, f, b.z), fmaf(st[r].acc[3].y, f, b.w));
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rows * 64; i += blockDim.x) {
    const int r = i >> 6, d = i & 63;
    float t = 0.f;
    if (WPS == 1) {
      for (int x = 0; x < warps; ++x) t += part[x][r][d];
    } else {
      for (int x = 0; x < slots; ++x) {
        const float w = slot_w[x];
        if (!slot_reads[x]) continue;                            // its parts hold no state
        float m = g.off_by_one > 0.f ? 0.f : -INFINITY;
#pragma unroll
        for (int y = 0; y < WPS; ++y) m = fmaxf(m, part[x * WPS + y][r][0]);
        float l = g.off_by_one > 0.f ? g.off_by_one * ex2f(-m) : 0.f, o = 0.f;
#pragma unroll
        for (int y = 0; y < WPS; ++y) {
          const float c = ex2f(part[x * WPS + y][r][0] - m);
          l = fmaf(part[x * WPS + y][r][1], c, l);
          o = fmaf(part[x * WPS + y][r][2 + d], c, o);
        }
        t = fmaf(o, w / l, t);
      }
    }
    if (ctas > 1) total[r][d] = t;
    else {
      const int gi = (row0 + r) / g.S, s = row0 + r - gi * g.S;
      out[n * g.os[0] + j * g.os[1] + (hk * g.G + gi) * g.os[2] + s * g.os[3] + d] = __float2bfloat16_rn(t);
    }
  }
  if (ctas > 1) {                                                // the first CTA adds the others' sums, in their order
    cluster_sync();
    if (rank == 0)
      for (int i = threadIdx.x; i < rows * 64; i += blockDim.x) {
        const int r = i >> 6, d = i & 63;
        float t = total[r][d];
        for (int x = 1; x < ctas; ++x) t += ld_dsmem(&total[r][d], x);
        const int gi = (row0 + r) / g.S, s = row0 + r - gi * g.S;
        out[n * g.os[0] + j * g.os[1] + (hk * g.G + gi) * g.os[2] + s * g.os[3] + d] = __float2bfloat16_rn(t);
      }
    cluster_sync();                                              // nobody leaves while its sums may be read
  }
}

// How the slots of an item are dealt out: warps per slot, CTAs per item (a cluster), warps per CTA (a multiple of wps).
//
// What counts is that all CTAs run at once (a second wave nearly doubles the time: one row, K = 8, 384 items 10.3 us, 480 16.9 unless four
// warps take two slots each: 15.4) and, within that, that as few steps as possible follow one another in a warp, and that an item is one CTA:
// a cluster costs ~0.6 us.  So: the first of these that fits one wave, from the shortest chain to the longest.
//   four warps a slot      K = 8, 100 items: 5.9 us in one CTA of 32 warps against 6.4 as two warps a slot and 7.7 as one.  Clusters of eight
//                          warps each start sooner where every CTA has an SM to itself (12 items: 4.3 against 5.0), and clusters of
//                          twelve or sixteen hold more than eight slots (K = 16, 64 items: 6.9 against 7.6 of a warp a slot)
//   two warps a slot       one CTA: K = 8, 148 items 7.0 against 7.4.  In clusters only for two rows, whose chain is the longer one
//                          (K = 16, 64 items: 7.7 against 8.6; one row 8.1 against 7.6), and for one row where a CTA cannot hold all slots
//   a warp a slot          one CTA if it holds them (K = 13, 148 items: 8.4 against 10.2 of two CTAs), else a cluster of two to four
//   two, three .. slots a warp, one CTA: the rounds r and waves w with the least w (r + 0.9).  The bytes take the same time however they are
//                          split; what differs is a round's latency (~3.4 us) in every wave, and a wave's start and merges (~3 us).  One
//                          row, K = 8, 1000 items: three rounds in one wave 25.5 us, two in two 30.9, one in three 29.9
// A CTA of a warp a slot has a multiple of four warps where that many still run at once, the last ones idle: the SM's quarters then have the same
// number of loads in flight (one row, K = 6, 384 items: eight warps 9.0 us, six 9.8; K = 3, 700 items: four 8.8, three 10.1; two rows, K = 5, 240
// items: eight 8.0, five 8.7).  Two rows keep an even number: six are 3 % faster than eight.
// Measured over rows 1, 2 x K 2 .. 32 x 148 .. 3000 items (caches from memory): within 0.3 % of the best of all splits on average (3.7 % above it with
// the first split of at most four warps a CTA beyond one wave, and 25 warps of 80 registers counted where 24 fit).  Two rows at
// 96 registers a thread instead of 128 fit more warps and lose 12 %: they spill.  Three and four rows are two pairs: 250 registers left
// 8 warps an SM (K = 8, 184 items 16.7 us as four rows, 14.2 as pairs).  An item's pairs are neighbours in the grid, so that the second reading
// of its K and V hits L2 however many items there are (K = 8, 1500 items, four rows 71 us; all first pairs before all second ones 84; as four rows 103).
struct DecodePlan { int wps, ctas, warps; };
DecodePlan decode_plan(long long items, int K, int rows, int sms) {
  const int cap4 = rows > 1 ? ROW_WARPS<2, 4> : ROW_WARPS<1, 4>, cap = rows > 1 ? ROW_WARPS<2, 1> : ROW_WARPS<1, 1>;
  const int sm_warps4 = warps_per_sm(rows > 1 ? ROW_REGS<2, 4> : ROW_REGS<1, 4>), sm_warps = warps_per_sm(rows > 1 ? ROW_REGS<2, 1> : ROW_REGS<1, 1>);
  if (rows > 1) items *= (rows + 1) / 2;
  DecodePlan plan = {0, 0, 0};
  auto take = [&](int wps, int ctas) {
    const int slots = (K + ctas - 1) / ctas, warps = slots * wps;
    // clusters leave some places empty: all of a cluster's CTAs have to find theirs in one group of SMs
    const int slack = ctas == 1 ? 0 : ctas < 5 ? 1 : ctas;
    if (ctas > 8 || (K + slots - 1) / slots != ctas || warps > (wps == 4 ? cap4 : cap)) return false;
    if (items * ctas * (16 + slack) > 16ll * sms * ((wps == 4 ? sm_warps4 : sm_warps) / warps)) return false;
    plan = {wps, ctas, warps};
    return true;
  };
  const int by2 = (K + 1) / 2, by3 = (K + 2) / 3, by4 = (K + 3) / 4;
  if (K > 6 && items * by2 <= sms && take(4, by2)) return plan;
  if (take(4, 1) || (K > 4 && (take(4, by3) || take(4, by4))) || take(2, 1)) return plan;
  if (rows > 1 && K > 8 && take(2, by4)) return plan;
  auto quartered = [&] {
    const int warps = (plan.warps + 3) & ~3;
    if ((rows == 1 || plan.warps % 2) && warps <= cap && items <= (long long)sms * (sm_warps / warps)) plan.warps = warps;
    return plan;
  };
  if (take(1, 1)) return quartered();
  if (K > 8 && (take(2, by4) || take(1, 2) || take(1, 3) || take(1, 4))) return plan;
  long long least = 0;
  for (int rounds = (K + cap - 1) / cap; rounds <= K; ++rounds) {
    const int warps = (K + rounds - 1) / rounds;
    const long long wave = (long long)sms * (sm_warps / warps), cost = (items + wave - 1) / wave * (10 * rounds + 9);
    if (least == 0 || cost < least) { least = cost; plan = {1, 1, warps}; }
    if (items <= wave) break;                                    // one wave: more rounds only take longer
  }
  return quartered();
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
    const DecodePlan plan = decode_plan(blocks, g.K, rows, sms);
    auto run = [&](auto kernel) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(blocks * plan.ctas * ((rows + 1) / 2))); cfg.blockDim = dim3((unsigned)(plan.warps * 32)); cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = 1;
      attr[1].id = cudaLaunchAttributeClusterDimension;
      attr[1].val.clusterDim.x = (unsigned)plan.ctas; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
      cfg.attrs = attr; cfg.numAttrs = plan.ctas > 1 ? 2 : 1;
      return (int)cudaLaunchKernelEx(&cfg, kernel, q, kc, vc, a.indices, a.weights, out, a.status, g, plan.ctas);
    };
    auto pick = [&](auto one, auto two, auto four) { return plan.wps == 1 ? run(one) : plan.wps == 2 ? run(two) : run(four); };
    if (rows <= 1) return pick(decode_rows_kernel<1, 1>, decode_rows_kernel<1, 2>, decode_rows_kernel<1, 4>);
    return pick(decode_rows_kernel<2, 1>, decode_rows_kernel<2, 2>, decode_rows_kernel<2, 4>);
  }
  int rc;
  if ((rc = make_tile_map_5d(&p.tm_k, a.k_cache, 64, 64, a.Hkv, a.C, a.N, a.k_stride[2], a.k_stride[3], a.k_stride[1], a.k_stride[0], 1, true))) return rc;
  if ((rc = make_tile_map_5d(&p.tm_v, a.v_cache, 64, 64, a.Hkv, a.C, a.N, a.v_stride[2], a.v_stride[3], a.v_stride[1], a.v_stride[0], 1, false))) return rc;
  if (rows <= 8) return launch_decode_r<8>(p, blocks, sms, stream);
  if (rows <= 16) return launch_decode_r<16>(p, blocks, sms, stream);
  return GCA_ERR_ALGO;
}

}  // namespace gca
