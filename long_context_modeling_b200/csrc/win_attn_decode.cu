// Sliding-window causal self-attention with ALiBi for a handful of new positions against the
// cached window (autoregressive decode): what the reference gets from flash-attn's
// flash_attn_with_kvcache(q, k, v, causal=True, window_size=(W, 0), alibi_slopes=m) at
// model/llama.py:684-688.  Per decoded token this reads 2 x (W + 1) x 128 bytes per (sequence, kv
// head) and layer: HBM-bound.
//
//   s[i, j] = scale * q_i . k_j  -  slope_h * (pos_i - j),   pos_i = T - Sq + i  (bottom-right aligned)
//   visible: pos_i - W <= j <= pos_i;   out_i = softmax_j(s[i, :]) V
//
// A CTA, or a cluster of them, per (sequence, kv head) and pair of rows; a warp takes sixteen keys at a time, straight from
// registers.  Two kernels, chosen at window_plan(): `win_once_kernel` where there are warps for all sixteens at once,
// `win_rounds_kernel` where several follow one another in a warp.  The warps' states and the CTAs' are merged in a fixed order:
// the result does not depend on scheduling.
//
// Bound: HBM for many items, else latency (launch, one round of loads, the merges).  Eight warps an item, one key at a time and
// multiply-adds took, us, one row: 512 keys, 4 items 6.9, now 4.8; 64 items 8.8, now 5.8; 384 items 13.3, now 12.7 (7.7 at the
// copy rate); two rows, 384 items 23.0, now 12.6.  With multiply-adds in the second kernel too (four keys a step) 13.9 and 13.9.  The same matrix instructions in the first kernel are slower (128 keys, 148
// items 4.0 us against 3.4): their chain is the longer one.
//
// RING form (decode of one position per sequence against a FULL window): the window buffer is a
// ring, the step's new K / V row arrives separately and replaces the oldest row.  With a
// device-side count c of rows written so far, the new row goes to physical row p = c mod T, and
// physical row j holds logical position (j - p - 1) mod T.  The new row is taken from its own operands
// and stored into row p; what a stream reads in row p itself, the oldest row or already the new one, is
// masked; every other row is read in place: the window never moves (shifting it costs a full read + write of the window per
// token and layer, more than the attention itself reads).
#include "gca_common.cuh"
#include "row_attn.cuh"
#include "sm100_ptx.cuh"

#include <algorithm>

namespace gca {

namespace {

using row_attn::ex2;
using row_attn::finite_max;
using row_attn::high;
using row_attn::load16;
using row_attn::low;

struct WinParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  const float* slopes;        // (Hq) or nullptr
  __nv_bfloat16* out;
  long long qs[3], os[3];     // strides of (n, head, row) in elements; the 64 head dims are contiguous
  long long ks[3], vs[3];     // strides of (n, kv head, position)
  int N, Hq, Hkv, G, Sq, T, window;
  float c2;                   // scale * log2(e)
  // ring form (else nullptr): the new position's rows by strides (n, kv head) and the count of rows written
  const __nv_bfloat16* knew;
  const __nv_bfloat16* vnew;
  const long long* ring;
  long long ns[2];
};

// Registers a thread and the most warps a CTA of the kernels has.
template <int R, bool ROUNDS> constexpr int WIN_REGS = R > 1 ? 128 : ROUNDS ? 80 : 64;
template <int R, bool ROUNDS> constexpr int WIN_WARPS = R > 1 ? 16 : ROUNDS ? 24 : 32;

template <int R> using WarpState = float[R][2 + 64];            // maximum, sum, 64 outputs of the rows

// The kernels' first row: one row's is blockIdx.y, which is 0 -- as a constant it makes the 80-register kernel spill more (384 items x 512 keys 11.73
// us, 11.62 so).
// The warps' states (and a cluster's CTAs') to the outputs, in a fixed order.
template <int R>
__device__ __forceinline__ void merge_and_store(const WinParams& p, WarpState<R>* part, WarpState<R>& total, int ctas, int rank, int n, int hk, int row0, int rows) {
  const int warps = blockDim.x >> 5;
  __syncthreads();
  auto store = [&](int r, int d, float l, float o) {
    const int gi = (row0 + r) / p.Sq, i = row0 + r - gi * p.Sq, h = hk * p.G + gi;
    p.out[n * p.os[0] + h * p.os[1] + i * p.os[2] + d] = __float2bfloat16_rn(p.T - p.Sq + i >= 0 ? o / l : 0.f);
  };
  for (int i = threadIdx.x; i < rows * 64; i += blockDim.x) {
    const int r = i >> 6, d = i & 63;
    float m = -INFINITY;
    for (int w = 0; w < warps; ++w) m = fmaxf(m, part[w][r][0]);
    const float mf = finite_max(m);
    float l = 0.f, o = 0.f;
    for (int w = 0; w < warps; ++w) {
      const float c = ex2(part[w][r][0] - mf);
      l = fmaf(part[w][r][1], c, l);
      o = fmaf(part[w][r][2 + d], c, o);
    }
    if (ctas == 1) store(r, d, l, o);
    else { total[r][2 + d] = o; if (d == 0) { total[r][0] = m; total[r][1] = l; } }
  }
  if (ctas > 1) {                                                // the first CTA merges the others' states, in their order
    sm100::cluster_sync();
    if (rank == 0)
      for (int i = threadIdx.x; i < rows * 64; i += blockDim.x) {
        const int r = i >> 6, d = i & 63;
        float m = total[r][0];
        for (int x = 1; x < ctas; ++x) m = fmaxf(m, sm100::ld_dsmem(&total[r][0], x));
        const float mf = finite_max(m);
        float l = 0.f, o = 0.f;
        for (int x = 0; x < ctas; ++x) {
          const float c = ex2(sm100::ld_dsmem(&total[r][0], x) - mf);
          l = fmaf(sm100::ld_dsmem(&total[r][1], x), c, l);
          o = fmaf(sm100::ld_dsmem(&total[r][2 + d], x), c, o);
        }
        store(r, d, l, o);
      }
    sm100::cluster_sync();                                       // nobody leaves while its state may be read
  }
}

// One warp for sixteen keys, in one round: latency counts.  A warp load covers FOUR key rows: 8 lanes x 16 bytes per 128-byte row; each 8-lane
// group has a stream of four keys, the streams are merged within the warp.  R rows of the kv head (blockIdx.x: which of its row pairs).  The
// ring's new row and the window's last row stand beside the sixteens, in the first warp: a window of 512 is 513 rows.
template <int R, bool RING>
__global__ void __maxnreg__((WIN_REGS<R, false>))
win_once_kernel(const WinParams p, int ctas) {
  __shared__ WarpState<R> part[WIN_WARPS<R, false>];
  __shared__ WarpState<R> total;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, sub = lane & 7, warps = blockDim.x >> 5;
  const int unit = blockIdx.x / ctas, rank = blockIdx.x - unit * ctas;
  const bool pairs = R > 1 && p.G * p.Sq > R;                    // three or four rows: an item's two pairs follow one another
  const int item = pairs ? unit >> 1 : unit, row0 = R == 1 ? blockIdx.y : pairs ? (unit & 1) * R : 0, rows = min(R, p.G * p.Sq - row0);
  const int n = item / p.Hkv, hk = item - n * p.Hkv;
  pdl_trigger();
  pdl_wait();
  const int last = p.T - 1;
  const int first = max(0, p.T - p.Sq - p.window);             // keys any row can see: [first, T)
  const __nv_bfloat16* kb = p.k + n * p.ks[0] + hk * p.ks[1] + sub * 8;
  const __nv_bfloat16* vb = p.v + n * p.vs[0] + hk * p.vs[1] + sub * 8;
  const long long written = RING ? *p.ring : 0;
  const int j0 = first + (rank * warps + warp) * 16 + grp;      // and 4, 8, 12 further on
  const __nv_bfloat16 *kp = kb + j0 * p.ks[2], *vp = vb + j0 * p.vs[2];
  uint4 kq[4], vq[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    kq[s] = vq[s] = make_uint4(0, 0, 0, 0);
    if (j0 + s * 4 < last) { kq[s] = load16(kp); vq[s] = load16(vp); }
    kp += 4 * p.ks[2]; vp += 4 * p.vs[2];
  }
  const bool extra = rank == 0 && warp == 0;                     // group 0 has the ring's new row, group 1 the last row
  uint4 kx = make_uint4(0, 0, 0, 0), vx = kx;
  if (extra && grp < 2) {
    if (RING && grp == 0) {
      kx = load16(p.knew + n * p.ns[0] + hk * p.ns[1] + sub * 8); vx = load16(p.vnew + n * p.ns[0] + hk * p.ns[1] + sub * 8);
    } else if (grp == 1) {
      kx = load16(kb + last * p.ks[2]); vx = load16(vb + last * p.vs[2]);
    }
  }
  uint4 qv[R];                                                   // this lane's 8 values of every row, the row's ALiBi slope (in log2 units) and position
  float slope[R];
  int pos[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int gi = (row0 + r) / p.Sq, i = row0 + r - gi * p.Sq, h = hk * p.G + gi;
    pos[r] = p.T - p.Sq + i;
    slope[r] = 0.f;
    qv[r] = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      slope[r] = p.slopes ? p.slopes[h] * GCA_LOG2E : 0.f;
      qv[r] = load16(p.q + n * p.qs[0] + h * p.qs[1] + i * p.qs[2] + sub * 8);
    }
  }
  // Ring: physical row `newest` is the new row's (the count stays below 2^32: caller's contract).  The linear form's newest row is the last one.
  const int newest = RING ? (int)((unsigned)written % (unsigned)p.T) : last;
  // how far key j lies behind row r's position, and whether the row sees it
  auto distance = [&](int r, int j) {
    const int d = (RING ? newest : pos[r]) - j;
    return RING && d < 0 ? d + p.T : d;
  };
  auto sees = [&](int d) { return RING ? d != 0 : d >= 0 && d <= p.window; };
  auto pair = [](uint32_t v) { return make_float2(low(v), high(v)); };
  auto splat = [](float v) { return make_float2(v, v); };
  auto dot = [&](int r, const uint4& k) {
    float2 t = __fmul2_rn(pair(qv[r].x), pair(k.x));
    t = __ffma2_rn(pair(qv[r].y), pair(k.y), t);
    t = __ffma2_rn(pair(qv[r].z), pair(k.z), t);
    t = __ffma2_rn(pair(qv[r].w), pair(k.w), t);
    return t.x + t.y;
  };
  float m[R], l[R];
  float2 acc[R][4];
  auto add = [&](int r, float w, const uint4& v, bool ok) {      // a masked row's values, whatever they are, count as zero
    acc[r][0] = __ffma2_rn(splat(w), pair(ok ? v.x : 0u), acc[r][0]); acc[r][1] = __ffma2_rn(splat(w), pair(ok ? v.y : 0u), acc[r][1]);
    acc[r][2] = __ffma2_rn(splat(w), pair(ok ? v.z : 0u), acc[r][2]); acc[r][3] = __ffma2_rn(splat(w), pair(ok ? v.w : 0u), acc[r][3]);
  };
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float sc[4], x = -INFINITY;
#pragma unroll
    for (int s = 0; s < 4; ++s) sc[s] = dot(r, kq[s]);
#pragma unroll
    for (int of = 1; of < 8; of <<= 1)
#pragma unroll
      for (int s = 0; s < 4; ++s) sc[s] += __shfl_xor_sync(0xffffffffu, sc[s], of);
    bool ok_x = false;
    if (extra) {                                                 // warp-uniform
      x = dot(r, kx);
#pragma unroll
      for (int of = 1; of < 8; of <<= 1) x += __shfl_xor_sync(0xffffffffu, x, of);
      const int d = RING && grp == 0 ? 0 : distance(r, last);
      ok_x = RING && grp == 0 ? true : grp == 1 && sees(d);
      x = ok_x ? fmaf(x, p.c2, -slope[r] * (float)d) : -INFINITY;
    }
    m[r] = x;
    bool ok[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int j = j0 + s * 4, d = distance(r, j);
      ok[s] = j < last && sees(d);
      sc[s] = ok[s] ? fmaf(sc[s], p.c2, -slope[r] * (float)d) : -INFINITY;
      m[r] = fmaxf(m[r], sc[s]);
    }
    m[r] = fmaxf(m[r], -INFINITY);                               // NaN is not a maximum, it stays in the sum
    const float mf = finite_max(m[r]);
    l[r] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[r][e] = splat(0.f);
    if (extra) { x = ex2(x - mf); l[r] = x; add(r, x, vx, ok_x); }
#pragma unroll
    for (int s = 0; s < 4; ++s) { sc[s] = ex2(sc[s] - mf); l[r] += sc[s]; add(r, sc[s], vq[s], ok[s]); }
  }
  if (RING && extra && grp == 0 && row0 == 0) {                  // over the oldest row, which nobody uses any more
    *reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(kb) + newest * p.ks[2]) = kx;
    *reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(vb) + newest * p.vs[2]) = vx;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {                                  // the four streams: one maximum, then plain sums
    float mw = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 8));
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 16));
    const float corr = ex2(m[r] - finite_max(mw));
    l[r] *= corr;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[r][e] = __fmul2_rn(acc[r][e], splat(corr));
#pragma unroll
    for (int of = 8; of <= 16; of <<= 1) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], of);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[r][e].x += __shfl_xor_sync(0xffffffffu, acc[r][e].x, of);
        acc[r][e].y += __shfl_xor_sync(0xffffffffu, acc[r][e].y, of);
      }
    }
    float* dst = part[warp][r];
    if (lane == 0) { dst[0] = mw; dst[1] = l[r]; }
    if (grp == 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(dst + 2 + sub * 8 + 2 * e) = acc[r][e];
    }
  }
  merge_and_store<R>(p, part, total, ctas, rank, n, hk, row0, rows);
}

// Several rounds of sixteen keys a warp: throughput counts, the next sixteen rows are on their way while these are worked on, on the tensor
// cores (row_attn.cuh).  The extra rows are a sixteen of the first warp's, before its others: a fifth round for them made a window of 512 a
// quarter longer.
template <int R, bool RING>
__global__ void __maxnreg__((WIN_REGS<R, true>))
win_rounds_kernel(const WinParams p, int) {                      // one CTA an item
  __shared__ WarpState<R> part[WIN_WARPS<R, true>];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warps = blockDim.x >> 5;
  const bool pairs = R > 1 && p.G * p.Sq > R;                    // three or four rows: an item's two pairs follow one another
  const unsigned item = pairs ? blockIdx.x >> 1 : blockIdx.x;
  const int row0 = R == 1 ? blockIdx.y : pairs ? (blockIdx.x & 1) * R : 0, rows = min(R, p.G * p.Sq - row0);
  const int n = item / p.Hkv, hk = item - n * p.Hkv;
  pdl_trigger();
  pdl_wait();
  const int first = max(0, p.T - p.Sq - p.window);             // keys any row can see: [first, T)
  // Sixteens of keys: [first, last) in order, dealt out over the warps, and one with the ring's new row and the window's last row
  const bool extra = RING || p.Sq == 1;
  const int last = extra ? p.T - 1 : p.T;
  const __nv_bfloat16* kb = p.k + n * p.ks[0] + hk * p.ks[1] + t * 8;
  const __nv_bfloat16* vb = p.v + n * p.vs[0] + hk * p.vs[1] + g * 8;
  const long long written = RING ? *p.ring : 0;
  uint4 kq[2][2], vq[4];
  const __nv_bfloat16 *kp = kb + (first + warp * 16 + g) * p.ks[2], *vp = vb + (first + warp * 16 + 2 * t) * p.vs[2];
  auto load_k = [&](int j0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = j0 + row_attn::key_of_k(lane, h);
      kq[h][0] = kq[h][1] = make_uint4(0, 0, 0, 0);
      if (j < last) { kq[h][0] = load16(kp + h * 8 * p.ks[2]); kq[h][1] = load16(kp + h * 8 * p.ks[2] + 32); }
    }
    kp += warps * 16 * p.ks[2];
  };
  auto load_v = [&](int j0) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int j = j0 + row_attn::key_of_v(lane, s);
      vq[s] = make_uint4(0, 0, 0, 0);
      if (j < last) vq[s] = load16(vp + ((s >> 1) * 8 + (s & 1)) * p.vs[2]);
    }
    vp += warps * 16 * p.vs[2];
  };
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const int span = warps * 16;
  int jb = first + warp * 16;                  // this warp's sixteen
  load_k(jb); load_v(jb);
  const bool has_extra = extra && warp == 0;                     // warp-uniform
  uint4 kx[2] = {zero, zero}, vx[2] = {zero, zero};
  if (has_extra) {
    const __nv_bfloat16* row = g == 1 ? kb + last * p.ks[2] : RING && g == 0 ? p.knew + n * p.ns[0] + hk * p.ns[1] + t * 8 : nullptr;
    if (row) { kx[0] = load16(row); kx[1] = load16(row + 32); }
    if (t == 0) {
      if (RING) vx[0] = load16(p.vnew + n * p.ns[0] + hk * p.ns[1] + g * 8);
      vx[1] = load16(vb + last * p.vs[2]);
    }
  }
  // the query rows, and of this lane's row the ALiBi slope (in log2 units) and position
  const __nv_bfloat16* qr[2] = {nullptr, nullptr};
  float slope = 0.f;
  int pos = 0, pos_of[2] = {0, 0};
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r < rows) {
      const int gi = (row0 + r) / p.Sq, i = row0 + r - gi * p.Sq, h = hk * p.G + gi;
      qr[r] = p.q + n * p.qs[0] + h * p.qs[1] + i * p.qs[2];
      pos_of[r] = p.T - p.Sq + i;
      if (R == 1 || (t & 1) == r) { slope = p.slopes ? p.slopes[h] * GCA_LOG2E : 0.f; pos = pos_of[r]; }
    }
  if (rows < R) pos_of[R - 1] = pos_of[0];
  const row_attn::Query q = row_attn::query<R>(qr[0], qr[1], lane);
  // Ring: physical row `newest` is the new row's (the count stays below 2^32: caller's contract).  The linear form's newest row is the last one.
  const int newest = RING ? (int)((unsigned)written % (unsigned)p.T) : last;
  row_attn::State st;
  row_attn::reset(st);
  // a dot product as a score: how far key j lies behind this lane's row, and whether the row sees it
  auto score = [&](float x, int j, bool there) {
    int d = (RING ? newest : pos) - j;
    if (RING && d < 0) d += p.T;
    const bool sees = there && (RING ? d != 0 : d >= 0 && d <= p.window);
    return sees ? fmaf(x, p.c2, -slope * (float)d) : -INFINITY;
  };
  // a key that the row does not see counts with zeros, whatever its row of V holds
  auto blank_v = [&](int j0, int row_pos) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int d = (RING ? newest : row_pos) - (j0 + row_attn::key_of_v(lane, s));
      if (RING ? d == 0 : d < 0 || d > p.window) vq[s] = make_uint4(0, 0, 0, 0);
    }
  };
  if (has_extra) {
    if (RING && row0 == 0) {                                     // the new row over the oldest one, which nobody uses any more
      if (g == 0) {
        __nv_bfloat16* kd = const_cast<__nv_bfloat16*>(kb) + newest * p.ks[2];
        *reinterpret_cast<uint4*>(kd) = kx[0]; *reinterpret_cast<uint4*>(kd + 32) = kx[1];
      }
      if (t == 0) *reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(vb) + newest * p.vs[2]) = vx[0];
    }
    float s[2];
    const uint4 k[2][2] = {{kx[0], kx[1]}, {zero, zero}}, v[4] = {vx[0], RING && newest == last ? zero : vx[1], zero, zero};
    row_attn::scores(q, k, s);
    s[0] = RING && g == 0 ? s[0] * p.c2 : score(s[0], last, g == 1);
    s[1] = -INFINITY;
    row_attn::accumulate<R>(st, s, v, lane);
  }
#pragma unroll 1
  for (; jb < last; jb += span) {
    float s[2];
    row_attn::scores(q, kq, s);
    load_k(jb + span);
#pragma unroll
    for (int h = 0; h < 2; ++h) { const int j = jb + row_attn::key_of_k(lane, h); s[h] = score(s[h], j, j < last); }
    if (RING || p.Sq > 1) blank_v(jb, pos_of[0]);
    if (!RING && R == 2 && pos_of[0] != pos_of[R - 1] &&
        ((jb + 15 > pos_of[0] && jb <= pos_of[R - 1]) || (jb + 15 >= pos_of[0] - p.window && jb < pos_of[R - 1] - p.window))) {
      // a row sees a key that the other does not: first the one's, then the other's, each into its own columns only (a weight of 0 times
      // an infinite value would not be nothing)
#pragma unroll 1
      for (int r = 0; r < 2; ++r) {
        float mine[2] = {(t & 1) == r ? s[0] : -INFINITY, (t & 1) == r ? s[1] : -INFINITY}, keep[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) { keep[i][0] = r ? st.acc[i][0] : st.acc[i][1]; keep[i][1] = r ? st.acc[i][2] : st.acc[i][3]; }
        if (r) { vp -= span * p.vs[2]; load_v(jb); blank_v(jb, pos_of[R - 1]); }
        row_attn::accumulate<R>(st, mine, vq, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (r) { st.acc[i][0] = keep[i][0]; st.acc[i][2] = keep[i][1]; }
          else { st.acc[i][1] = keep[i][0]; st.acc[i][3] = keep[i][1]; }
        }
      }
    } else {
      row_attn::accumulate<R>(st, s, vq, lane);
    }
    load_v(jb + span);
  }
  float o[R][8];
  row_attn::finish<R>(st, o);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float* dst = part[warp][r];
    if (lane == r) { dst[0] = st.m; dst[1] = st.l; }            // lane r = row r's
    if (t == 0) {
#pragma unroll
      for (int e = 0; e < 8; e += 2) *reinterpret_cast<float2*>(dst + 2 + g * 8 + e) = make_float2(o[r][e], o[r][e + 1]);
    }
  }
  merge_and_store<R>(p, part, part[0], 1, 0, n, hk, row0, rows);
}

// Which kernel, and how the sixteens of an item (a kv head's row pair) are dealt out over warps and CTAs (a cluster).  All CTAs have to run at
// once, and as few rounds as possible to follow one another.  So, the first of these that fits one wave (one row, us):
//   once, one CTA        256 keys, 148 items 5.0 (two rounds 5.8), 256 items 6.8 (7.9)
//   once, a cluster      of four, three or two CTAs where two have an SM to themselves: 640 keys, 4 items 4.6 (two rounds in one CTA 6.0)
//   rounds               two, three .. in one CTA, the rounds r and waves w with the least w (r + 1.5): 512 keys, 256 items three of eleven warps
//                        9.8 (four of eight 10.9), 384 items four of eight 12.7, 640 items eight of four 18.4 (seven of five in two waves 24.1)
// Over one and two rows x 64 .. 640 keys x 148 .. 3000 items (caches from memory) 0.1 % above the best of these splits on average (3.5 % with the
// first split of at most four warps a CTA beyond one wave, and 25 warps of 80 registers counted where 24 fit).  Two rows at
// 80 registers a thread fit more warps and lose 10 % where both fit (512 keys, 148 items 8.2 against 7.4).
// Three and four rows are two pairs, neighbours in the grid: the second reading of an item's window hits L2 (512 keys, 1500 items, four rows
// 56 us; all first pairs before all second ones 70).
struct WindowPlan { int ctas, warps; bool rounds; };
WindowPlan window_plan(long long items, int keys, int rows, int sms) {
  if (rows > 1) items *= (rows + 1) / 2;
  const int cap = rows > 1 ? WIN_WARPS<2, true> : WIN_WARPS<1, true>, cap_once = rows > 1 ? WIN_WARPS<2, false> : WIN_WARPS<1, false>;
  const int sm_warps = warps_per_sm(rows > 1 ? WIN_REGS<2, true> : WIN_REGS<1, true>);
  const int sm_warps_once = warps_per_sm(rows > 1 ? WIN_REGS<2, false> : WIN_REGS<1, false>);
  auto fits_once = [&](int ctas, int warps) { return warps <= cap_once && items * ctas <= (long long)sms * (sm_warps_once / warps); };
  const int sixteens = std::max(1, (keys + 15) / 16);
  if (fits_once(1, sixteens)) return {1, sixteens, false};
  for (int ctas = 4; ctas > 1; --ctas) {
    const int warps = (sixteens + ctas - 1) / ctas;
    if (2 * items * ctas <= sms && fits_once(ctas, warps)) return {ctas, warps, false};
  }
  WindowPlan plan = {1, std::min(cap, sixteens), true};
  long long least = 0;
  for (int rounds = std::max(2, (sixteens + cap - 1) / cap); rounds <= sixteens; ++rounds) {
    const int warps = (sixteens + rounds - 1) / rounds;
    const long long wave = (long long)sms * (sm_warps / warps), cost = (items + wave - 1) / wave * (2 * rounds + 3);
    if (least == 0 || cost < least) { least = cost; plan.warps = warps; }
    if (items <= wave) break;                                    // one wave: more rounds only take longer
  }
  return plan;
}

// The cached window of one decode step, moved on IN PLACE: every (sequence, head) block of T rows drops
// its oldest row and takes the new position's row at the end.  One CTA owns one block of K or V,
// reads it whole into registers (T <= 16 x 256 rows of 128 bytes... 16 bytes per thread and pass),
// synchronises, and writes it back one row down: no second buffer, no concatenation, 2 x T x 128 bytes of
// traffic per block (the torch.cat + copy it replaces moves twice that through slower kernels).
constexpr int SHIFT_THREADS = 256, SHIFT_MAX_VEC = 20;        // 16-byte vectors per thread: blocks of up to 640 rows
__global__ void __launch_bounds__(SHIFT_THREADS)
window_shift_append_kernel(__nv_bfloat16* __restrict__ kwin, __nv_bfloat16* __restrict__ vwin, const __nv_bfloat16* __restrict__ knew,
                           const __nv_bfloat16* __restrict__ vnew, int H, int T, long long ws0, long long ws1, long long ns0,
                           long long ns1) {
  const bool is_v = blockIdx.y != 0;
  const int n = blockIdx.x / H, h = blockIdx.x - n * H;
  uint4* win = reinterpret_cast<uint4*>((is_v ? vwin : kwin) + n * ws0 + h * ws1);     // T rows x 8 vectors, contiguous
  const uint4* fresh = reinterpret_cast<const uint4*>((is_v ? vnew : knew) + n * ns0 + h * ns1);
  const int total = T * 8;                        // vectors in the block
  uint4 r[SHIFT_MAX_VEC];
#pragma unroll
  for (int i = 0; i < SHIFT_MAX_VEC; ++i) {
    const int v = threadIdx.x + i * SHIFT_THREADS + 8;          // the vector one ROW further on
    if (v < total) r[i] = win[v];
    else if (v < total + 8) r[i] = fresh[v - total];            // the last row comes from the new position
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SHIFT_MAX_VEC; ++i) {
    const int v = threadIdx.x + i * SHIFT_THREADS;
    if (v < total) win[v] = r[i];
  }
}

}  // namespace

int launch_window_shift_append(const WindowAppendArgs& a, cudaStream_t stream) {
  if (a.T * 8 > SHIFT_THREADS * SHIFT_MAX_VEC) return GCA_ERR_SHAPE;
  const dim3 grid((unsigned)(a.N * a.H), 2);
  if (grid.x == 0) return 0;
  window_shift_append_kernel<<<grid, SHIFT_THREADS, 0, stream>>>((__nv_bfloat16*)a.k_window, (__nv_bfloat16*)a.v_window,
                                                                  (const __nv_bfloat16*)a.k_new, (const __nv_bfloat16*)a.v_new, a.H, a.T,
                                                                  a.window_stride[0], a.window_stride[1], a.new_stride[0], a.new_stride[1]);
  return (int)cudaGetLastError();
}

static int launch_window(const WindowDecodeArgs& a, const WindowRingDecodeArgs* ring, int sms, cudaStream_t stream) {
  WinParams p;
  p.knew = p.vnew = nullptr; p.ring = nullptr; p.ns[0] = p.ns[1] = 0;
  if (ring) {
    p.knew = (const __nv_bfloat16*)ring->k_new; p.vnew = (const __nv_bfloat16*)ring->v_new;
    p.ring = (const long long*)ring->rows_written; p.ns[0] = ring->new_stride[0]; p.ns[1] = ring->new_stride[1];
  }
  p.q = (const __nv_bfloat16*)a.q; p.k = (const __nv_bfloat16*)a.k; p.v = (const __nv_bfloat16*)a.v;
  p.slopes = a.alibi_slopes; p.out = (__nv_bfloat16*)a.out;
  for (int i = 0; i < 3; ++i) { p.qs[i] = a.q_stride[i]; p.os[i] = a.o_stride[i]; p.ks[i] = a.k_stride[i]; p.vs[i] = a.v_stride[i]; }
  p.N = a.N; p.Hq = a.Hq; p.Hkv = a.Hkv; p.G = a.Hq / a.Hkv; p.Sq = a.Sq; p.T = a.T; p.window = a.window;
  p.c2 = a.sm_scale * GCA_LOG2E;
  const int rows = p.G * a.Sq, items = a.N * a.Hkv;
  if (items == 0) return 0;
  if (rows > 4) return GCA_ERR_SHAPE;
  const WindowPlan plan = window_plan(items, p.T - (ring || a.Sq == 1 ? 1 : 0) - std::max(0, p.T - p.Sq - p.window), rows, sms);
  auto run = [&](auto kernel) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items * plan.ctas * ((rows + 1) / 2))); cfg.blockDim = dim3((unsigned)(plan.warps * 32)); cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)plan.ctas; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = plan.ctas > 1 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, p, plan.ctas);
  };
  auto form = [&](auto once, auto rounds) { return plan.rounds ? run(rounds) : run(once); };
  if (ring)                                        // one new position: G rows per kv head
    return rows <= 1 ? form(win_once_kernel<1, true>, win_rounds_kernel<1, true>) : form(win_once_kernel<2, true>, win_rounds_kernel<2, true>);
  return rows <= 1 ? form(win_once_kernel<1, false>, win_rounds_kernel<1, false>) : form(win_once_kernel<2, false>, win_rounds_kernel<2, false>);
}

int launch_window_decode(const WindowDecodeArgs& a, int sms, cudaStream_t stream) { return launch_window(a, nullptr, sms, stream); }

int launch_window_ring_decode(const WindowRingDecodeArgs& a, int sms, cudaStream_t stream) { return launch_window(a.attn, &a, sms, stream); }

}  // namespace gca
