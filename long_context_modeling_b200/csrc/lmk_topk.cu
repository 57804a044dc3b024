// Landmark scoring + causal chunk mask + top-k + retrieval weights.
//
// The cached landmarks (E rows of D bf16 values) are streamed once.  One warp scores one
// landmark row at a time: the row is cut in 8-element (16-byte) pieces, lane l owns pieces
// l, l+32, l+64, ... so every load instruction of the warp covers 512 contiguous bytes.
// The float32 dot product is accumulated in a FIXED order (pieces in increasing order inside
// a lane, then a butterfly over the lanes), which makes every score -- and therefore every
// selected index -- independent of grid size, split count and GPU count.
//
// Candidates are 64-bit keys  orderable(score) << 32 | (0xFFFFFFFF - global_index):  a
// larger key is a better candidate, equal scores resolve to the lower index, and merging
// lists from warps, blocks or GPUs is a plain integer top-k.  Key 0 means "empty".
//
// Each warp keeps its running top-K per query row as a sorted list spread over its lanes
// (lane i holds the i-th best).  Blocks write their lists to a scratch buffer; a second,
// tiny kernel merges the lists of all blocks of a row and emits indices, noise-free scores,
// softmax weights and the number of valid slots.
#include <algorithm>

#include "lmk_common.cuh"
#include "sm100_ptx.cuh"

namespace gca {
// lmk_tc_sm100.cu: many query rows per sequence
bool lmk_screen_applies(const LmkTopkArgs& a);
size_t lmk_screen_workspace_bytes(const LmkTopkArgs& a, int sms);
int launch_lmk_screen(const LmkTopkArgs& a, void* scratch, int sms, const FinalParams& fin, cudaStream_t stream);
}  // namespace gca

namespace gca {

namespace {

constexpr int SCAN_WARPS = 8;
struct ScanParams {
  const __nv_bfloat16* lq;
  const __nv_bfloat16* lk;
  const float* noise;
  unsigned long long* part;     // (rows, splits, K)
  long long qbs, qrs, kbs, krs;
  long long q_pos0, e_base;
  int N, Cq, E, D, K, H;
  int splits, e_per_split;
  int score_round;
  float scale;
};

constexpr int BATCH = 128;
// Merge a batch of 128 scores (o[i]: id id0 + 32 i + lane; orderable, 0 = none; all ids above those of the list) into a list of K keys held one per lane;
// `kth` is the list's K-th key.  Fewer than K that beat the list's K-th score are inserted, one after the other; K or more, and the K best come out
// by K warp-wide maxima of the 32-bit scores: whoever holds the maximum strikes it out and notes its key, which is all that the next round waits for (with
// the owner found by votes and its key shuffled to its place a round takes more than twice as long, with a vote on how many hold it nearly twice).
// Equal scores are struck out together: more struck out than rounds, and it is done over again with a second maximum a round, which finds the lowest
// id; at once where scores are rounded to 16 bits (`often_equal`).  K rounds from the third of a batch on cost 32 x 7,200 landmarks of 1,024, per
// head, K = 32 119 us (now 90), 32 x 7,200 of 768 93 (69), 4 x 37,000 57.6 (47.4), K = 16 45.2 (43.3).
__device__ __forceinline__ void select_batch(unsigned long long& mine, unsigned long long& kth, const unsigned o[4], unsigned id0, int K, int lane,
                                             bool often_equal, unsigned long long* note) {
  const unsigned th = (unsigned)(kth >> 32);                 // 0 while the list is not full
  unsigned b[4];
  int found = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) { b[i] = __ballot_sync(0xffffffffu, o[i] > th); found += __popc(b[i]); }
  if (found == 0) return;
  if (found < max(K, 3)) {                                   // lower ids first; what the first ones push below the K-th place stays there
#pragma unroll
    for (int i = 0; i < 4; ++i)
      for (unsigned m = b[i]; m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        list_insert(mine, ((unsigned long long)__shfl_sync(0xffffffffu, o[i], src) << 32) | (0xffffffffu - (id0 + 32 * i + src)), lane);
      }
    kth = __shfl_sync(0xffffffffu, mine, K - 1);
    return;
  }
  unsigned r = (unsigned)(mine >> 32), v[4] = {o[0], o[1], o[2], o[3]};
  const unsigned first = 0xffffffffu - (id0 + lane);
  auto highest = [&] { return __reduce_max_sync(0xffffffffu, max(max(max(r, v[0]), max(v[1], v[2])), v[3])); };
  int k = 0, struck = often_equal;
  for (; k < K && !often_equal; ++k) {
    const unsigned m = highest();
    if (m == 0u) break;
    unsigned low = (unsigned)mine;
    bool hit = r == m;
    if (hit) { r = 0u; ++struck; }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (v[i] == m) { v[i] = 0u; low = first - 32 * i; hit = true; ++struck; }
    if (hit) note[k] = ((unsigned long long)m << 32) | low;
  }
  if (__reduce_add_sync(0xffffffffu, struck) != k) {
    __syncwarp();
    r = (unsigned)(mine >> 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = o[i];
#pragma unroll 1
    for (k = 0; k < K; ++k) {
      const unsigned m = highest();
      if (m == 0u) break;
      unsigned low = 0u;                                     // ~id of this lane's first with that score
#pragma unroll
      for (int i = 3; i >= 0; --i)
        if (v[i] == m) low = first - 32 * i;
      if (r == m) low = (unsigned)mine;
      const unsigned lowest = __reduce_max_sync(0xffffffffu, low);
      if (low != lowest) continue;
      note[k] = ((unsigned long long)m << 32) | low;
      if (r == m) r = 0u;
      else
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (low == first - 32 * i) v[i] = 0u;
    }
  }
  __syncwarp();
  mine = lane < k ? note[lane] : 0ull;
  __syncwarp();
  kth = __shfl_sync(0xffffffffu, mine, K - 1);
}

// ---------------------------------------------------------------------------------------------
// One query row (a decode step), or one row and head at a time: the landmarks are streamed once, HBM-bound.
//
// Every lane copies the 16-byte pieces it will need itself to shared memory (cp.async), RING rows ahead of the
// arithmetic, so 196 KB per SM are on their way without a register or a barrier.  Scores of 128 rows at a time go to shared
// memory; list l (one per head, or the only one) is kept by warp l % 16, which merges
// the 128 scores into it (select_batch): one list per block instead of one per warp to merge at the end, and
// no list code in the scoring loop (per head it was 12 lists in every warp, each with a serial insertion: 60 us for
// 2 x 16,411 landmarks, now 14.8 with its merge; 262,144 landmarks, one list: 66.2 us = 6.1 TB/s with its
// merge).
constexpr int SPLIT_ROWS = 64, STREAM_WARPS = 16;                // rows that a block takes at least
template <int NP> constexpr int RING_ROWS = NP > 3 ? 6 : 8;       // 196 KB per SM
template <int NP> constexpr int ROWS_AT_ONCE = NP > 3 ? 2 : 4;    // of a warp

// One step of the butterfly over the lanes for two rows at a time: lanes whose bit `of` is clear go on with the sum of row a, the others with
// that of row b.  The same sums as a step for each (a sum of two does not depend on their order) for half the shuffles.
__device__ __forceinline__ float fold_rows(float a, float b, int of, int lane) {
  const bool up = lane & of;
  return (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, of);
}

// The K best of up to 32 descending lists, lane l at the head of list l: K times the best head, found by a warp-wide maximum, moves on.
// `at(i)`: this lane's list's entry i (0 past the end of a short list); lanes without a list pass has = false.
template <class At>
__device__ __forceinline__ unsigned long long merge_heads(int K, bool has, int lane, At at) {
  unsigned long long head = has ? at(0) : 0ull, next = has && K > 1 ? at(1) : 0ull, mine = 0ull;
  int taken = 1;
  for (int i = 0; i < K; ++i) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(head >> 32));
    if (hi == 0u) break;
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(head >> 32) == hi ? (unsigned)head : 0u);
    const unsigned long long best = ((unsigned long long)hi << 32) | lo;
    if (lane == i) mine = best;
    if (head == best) { head = next; ++taken; next = taken < K ? at(taken) : 0ull; }
  }
  return mine;
}
__device__ __forceinline__ unsigned long long ld_dsmem_u64(const unsigned long long* p, int rank) {       // the same variable in another CTA of the cluster
  unsigned long long v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.u64 %0, [a];\n\t}" : "=l"(v) : "r"(sm100::smem_u32(p)), "r"(rank) : "memory");
  return v;
}

// FUSED: the blocks of a row are a cluster, and the first one merges their lists and writes the row's outputs: no lists in memory, no
// second launch.  When, is said at fused().
template <int NP, bool PER_HEAD, bool FUSED>
__global__ void __launch_bounds__(STREAM_WARPS * 32, 1)
lmk_stream_kernel(ScanParams p, FinalParams fin) {
  constexpr int RING = RING_ROWS<NP>, U = ROWS_AT_ONCE<NP>, NL = PER_HEAD ? NP * 4 : 1, MINE = (NL + STREAM_WARPS - 1) / STREAM_WARPS, ROW_BYTES = NP * 512;
  extern __shared__ __align__(16) unsigned char ring_all[];            // [STREAM_WARPS][RING][ROW_BYTES]
  // A store's four heads in banks of their own (2 x 16,411 landmarks 15.2 -> 14.7 us).  The arrays stay a multiple of 128 bytes: the ring behind them would
  // not lie on the lines that are copied into it otherwise (262,144 landmarks, one list: 64.9 -> 67.5).
  constexpr int PITCH = PER_HEAD ? BATCH + 4 : BATCH;
  static_assert(2 * NL * PITCH * 4 % 128 == 0, "alignment of the ring");
  __shared__ float score[2][NL][PITCH];
  __shared__ unsigned long long note[NL < STREAM_WARPS ? NL : STREAM_WARPS][MAXK];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x, t0 = blockIdx.y, n = blockIdx.z;
  const int pieces = p.D >> 3;
  unsigned char* ring = ring_all + warp * RING * ROW_BYTES + lane * 16;
  const int e_lo = split * p.e_per_split;
  // the causal mask is a limit on the landmark id
  const long long seen = p.q_pos0 + t0 - p.e_base;
  const int e_hi = (int)max((long long)e_lo, min((long long)min(p.E, e_lo + p.e_per_split), seen));
  const __nv_bfloat16* kb = p.lk + n * p.kbs + lane * 8;
  // NP = ceil(D / 256): only a lane's last piece can be absent.  Nothing is ever copied to its place, which holds zeros.
  const bool last_piece = lane + 32 * (NP - 1) < pieces;
  if (!last_piece)
#pragma unroll
    for (int r = 0; r < RING; ++r) *reinterpret_cast<uint4*>(ring + r * ROW_BYTES + (NP - 1) * 512) = make_uint4(0, 0, 0, 0);
  // this warp's i-th row is e_lo + 16 i + warp; rows are asked for in order, two at a time
  const __nv_bfloat16* next_src = kb + (long long)(e_lo + warp) * p.krs;
  const long long src_step = p.krs * STREAM_WARPS;
  int next_e = e_lo + warp;
  auto fetch = [&](int slot) {                                // into the ring's places slot and slot + 1
    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + slot * ROW_BYTES);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (next_e < e_hi)
#pragma unroll
        for (int pp = 0; pp < NP; ++pp)
          if (pp + 1 < NP || last_piece)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + u * ROW_BYTES + pp * 512), "l"(next_src + pp * 256) : "memory");
      next_e += STREAM_WARPS;
      next_src += src_step;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_wait();
#pragma unroll
  for (int i = 0; i < RING; i += 2) fetch(i);
  float qf[NP][8];
#pragma unroll
  for (int pp = 0; pp < NP; ++pp) {
    const int c = lane + 32 * pp;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (c < pieces) v = *reinterpret_cast<const uint4*>(p.lq + n * p.qbs + (long long)t0 * p.qrs + c * 8);
    unpack8(v, qf[pp]);
  }
  unsigned long long mine[MINE], kth[MINE];
#pragma unroll
  for (int x = 0; x < MINE; ++x) mine[x] = kth[x] = 0ull;

  const int batches = (e_hi - e_lo + BATCH - 1) / BATCH;
  int slot = 0;
  for (int b = 0; b < batches; ++b) {
    float (*sc)[PITCH] = score[b & 1];
#pragma unroll
    for (int i = 0; i < BATCH / STREAM_WARPS; i += U) {
      if (e_lo + b * BATCH + i * STREAM_WARPS >= e_hi) break;
      constexpr int X = PER_HEAD ? NP : 1;
      float2 acc[U / 2][X];                                  // of two rows
#pragma unroll
      for (int u = 0; u < U; u += 2) {
        asm volatile("cp.async.wait_group %0;" ::"n"(RING / 2 - 1) : "memory");     // a lane reads only what it copied itself
#pragma unroll
        for (int x = 0; x < X; ++x) acc[u / 2][x] = make_float2(0.f, 0.f);
#pragma unroll
        for (int pp = 0; pp < NP; ++pp) {                    // absent pieces add 0 * 0: the sums never are -0
          const unsigned char* at = ring + (slot + u) * ROW_BYTES + pp * 512;
          float k0[8], k1[8];
          unpack8(*reinterpret_cast<const uint4*>(at), k0);
          unpack8(*reinterpret_cast<const uint4*>(at + ROW_BYTES), k1);
          float2& s = acc[u / 2][PER_HEAD ? pp : 0];
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) s = __ffma2_rn(make_float2(qf[pp][jj], qf[pp][jj]), make_float2(k0[jj], k1[jj]), s);
        }
        fetch(slot + u);
      }
      if ((slot += U) == RING) slot = 0;
      constexpr int TOP = PER_HEAD ? 4 : 16;                 // the butterfly starts at this distance
      float sum[X];
      int row = 0;                                           // of the U: the one whose score this lane ends up with
#pragma unroll
      for (int x = 0; x < X; ++x) {
        if (U == 4) {
          const float s0 = fold_rows(acc[0][x].x, acc[U / 2 - 1][x].x, TOP, lane), s1 = fold_rows(acc[0][x].y, acc[U / 2 - 1][x].y, TOP, lane);
          sum[x] = fold_rows(s0, s1, TOP / 2, lane);
          row = (lane & TOP ? 2 : 0) + (lane & (TOP / 2) ? 1 : 0);
        } else {
          sum[x] = fold_rows(acc[0][x].x, acc[0][x].y, TOP, lane);
          row = lane & TOP ? 1 : 0;
        }
#pragma unroll
        for (int of = U == 4 ? TOP / 4 : TOP / 2; of > 0; of >>= 1) sum[x] += __shfl_xor_sync(0xffffffffu, sum[x], of);
        sum[x] = p.score_round ? round_bf16(round_bf16(sum[x]) * p.scale) : sum[x] * p.scale;
      }
      if ((lane & (U == 4 ? TOP / 4 : TOP / 2) * 2 - 1) == 0)
#pragma unroll
        for (int x = 0; x < X; ++x) sc[PER_HEAD ? x * 4 + (lane >> 3) : 0][(i + row) * STREAM_WARPS + warp] = sum[x];
    }
    __syncthreads();
    const int e0 = e_lo + b * BATCH + lane;
#pragma unroll
    for (int x = 0; x < MINE; ++x) {
      const int l = warp + x * STREAM_WARPS;
      if (l >= NL || (PER_HEAD && l >= p.H)) continue;
      unsigned o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float s = sc[l][lane + 32 * i];
        if (p.noise && e0 + 32 * i < e_hi) s += p.noise[((long long)n * p.Cq + t0) * p.E + e0 + 32 * i];
        o[i] = e0 + 32 * i < e_hi ? orderable(s) : 0u;
      }
      select_batch(mine[x], kth[x], o, (unsigned)(p.e_base + e_lo + b * BATCH), p.K, lane, p.score_round != 0, note[warp]);
    }
  }
  if constexpr (FUSED) {
    __shared__ unsigned long long lists[NL][MAXK];
#pragma unroll
    for (int x = 0; x < MINE; ++x)
      if (warp + x * STREAM_WARPS < NL) lists[warp + x * STREAM_WARPS][lane] = mine[x];
    sm100::cluster_sync();
    if (split == 0) {
#pragma unroll 1
      for (int l = warp; l < NL && (!PER_HEAD || l < p.H); l += STREAM_WARPS) {
        const unsigned long long best = merge_heads(p.K, lane < p.splits, lane, [&](int i) { return ld_dsmem_u64(&lists[l][i], lane); });
        emit_row(fin, ((long long)n * p.Cq + t0) * p.H + l, best, lane);
      }
    }
    sm100::cluster_sync();                                     // nobody leaves while its lists may be read
  } else {
#pragma unroll
    for (int x = 0; x < MINE; ++x) {
      const int l = warp + x * STREAM_WARPS;
      if (l >= NL || (PER_HEAD && l >= p.H)) continue;
      const long long row = ((long long)n * p.Cq + t0) * p.H + l;
      if (lane < p.K) p.part[(row * p.splits + split) * p.K + lane] = mine[x];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// A few query rows per sequence (TQ per block): one warp scores one landmark row against all of them.
// NP: pieces per lane (D <= 256*NP).
template <int NP, int TQ>
__global__ void __launch_bounds__(SCAN_WARPS * 32)
lmk_scan_kernel(ScanParams p) {
  __shared__ unsigned long long sL[SCAN_WARPS][TQ][MAXK];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x, t0 = blockIdx.y * TQ, n = blockIdx.z;
  const int pieces = p.D >> 3;

  float qf[TQ][NP][8];
#pragma unroll
  for (int t = 0; t < TQ; ++t)
#pragma unroll
    for (int pp = 0; pp < NP; ++pp) {
      const int c = lane + 32 * pp;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (c < pieces && t0 + t < p.Cq)
        v = *reinterpret_cast<const uint4*>(p.lq + n * p.qbs + (long long)(t0 + t) * p.qrs + c * 8);
      unpack8(v, qf[t][pp]);
    }

  unsigned long long mine[TQ];
  // Admission test: a candidate enters a full list only if its score beats the list's K-th
  // score (rows arrive in increasing index order inside a warp, so an equal score loses the
  // tie; scores are never -0).  NaN while the list is not full: "!(s <= NaN)" admits everything.
  float thr_s[TQ];
#pragma unroll
  for (int l = 0; l < TQ; ++l) { mine[l] = 0ull; thr_s[l] = __int_as_float(0x7fc00000); }

  const int e_lo = split * p.e_per_split;
  const int e_hi = min(p.E, e_lo + p.e_per_split);
  const __nv_bfloat16* kb = p.lk + n * p.kbs;
  // the last query row of the tile sees the most chunks: rows past that limit are skipped
  const long long tile_limit = p.q_pos0 + min(t0 + TQ, p.Cq) - 1;
  constexpr int U = 2;                                // landmark rows in flight per warp iteration

  for (int e = e_lo + warp; e < e_hi; e += U * SCAN_WARPS) {
    uint4 kv[U][NP];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int eu = e + u * SCAN_WARPS;
#pragma unroll
      for (int pp = 0; pp < NP; ++pp) {
        const int c = lane + 32 * pp;
        kv[u][pp] = make_uint4(0, 0, 0, 0);
        if (eu < e_hi && c < pieces && p.e_base + eu < tile_limit)
          kv[u][pp] = *reinterpret_cast<const uint4*>(kb + (long long)eu * p.krs + c * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int eu = e + u * SCAN_WARPS;
      const long long eg = p.e_base + eu;
      if (eu >= e_hi || eg >= tile_limit) continue;     // warp-uniform
      float kf[NP][8];
#pragma unroll
      for (int pp = 0; pp < NP; ++pp) unpack8(kv[u][pp], kf[pp]);
#pragma unroll
      for (int t = 0; t < TQ; ++t) {
        float acc = 0.f;
#pragma unroll
        for (int pp = 0; pp < NP; ++pp)
          if (lane + 32 * pp < pieces) {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) acc = fmaf(qf[t][pp][jj], kf[pp][jj], acc);
          }
#pragma unroll
        for (int of = 16; of > 0; of >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, of);
        float s = p.score_round ? round_bf16(round_bf16(acc) * p.scale) : acc * p.scale;
        const int row = t0 + t;
        const bool vis = row < p.Cq && eg < p.q_pos0 + row;
        if (p.noise && vis) s += p.noise[((long long)n * p.Cq + row) * p.E + eu];
        if (vis && !(s <= thr_s[t])) {
          list_insert(mine[t], make_key(s, (unsigned)eg), lane);
          const unsigned long long kth = __shfl_sync(0xffffffffu, mine[t], p.K - 1);
          if (kth != 0ull) thr_s[t] = from_orderable((unsigned)(kth >> 32));
        }
      }
    }
  }

  // merge the 8 per-warp lists of every row of the tile; list l is merged by warp l % 8
#pragma unroll
  for (int l = 0; l < TQ; ++l)
    if (lane < p.K) sL[warp][l][lane] = mine[l];
  __syncthreads();
#pragma unroll
  for (int l = 0; l < TQ; ++l) {
    if ((l % SCAN_WARPS) != warp) continue;
    if (t0 + l >= p.Cq) continue;
    const long long row = (long long)n * p.Cq + t0 + l;
    unsigned long long m = 0ull, th = 0ull;
    for (int w = 0; w < SCAN_WARPS; ++w)
      for (int i = 0; i < p.K; ++i) {
        const unsigned long long key = sL[w][l][i];
        if (key <= th) break;                              // lists are descending
        list_insert(m, key, lane);
        th = __shfl_sync(0xffffffffu, m, p.K - 1);
      }
    if (lane < p.K) p.part[(row * p.splits + split) * p.K + lane] = m;
  }
}

constexpr int FIN_WARPS = 8;

// The merge of one row's P candidates (src) by one block of FIN_WARPS warps (sL: FIN_WARPS x MAXK
// keys of shared memory), and the decoded outputs of the row.
__device__ void finalize_row(const FinalParams& p, long long row, const unsigned long long* src,
                             unsigned long long (*sL)[MAXK]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // each warp merges a contiguous share of the candidates
  const int per = (p.P + FIN_WARPS - 1) / FIN_WARPS;
  const int lo = warp * per, hi = min(p.P, lo + per);
  unsigned long long m = 0ull, th = 0ull;
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const unsigned long long mykey = (i0 + lane < hi) ? __ldcg(src + i0 + lane) : 0ull;   // may have been written by another GPU
    unsigned pending = __ballot_sync(0xffffffffu, mykey > th);
    while (pending) {
      const int srcl = __ffs(pending) - 1;
      pending &= pending - 1;
      const unsigned long long key = __shfl_sync(0xffffffffu, mykey, srcl);
      if (key > th) {
        list_insert(m, key, lane);
        th = __shfl_sync(0xffffffffu, m, p.K - 1);
      }
    }
  }
  if (lane < p.K) sL[warp][lane] = m;
  __syncthreads();
  if (warp != 0) return;
  m = 0ull; th = 0ull;
  for (int w = 0; w < FIN_WARPS; ++w)
    for (int i = 0; i < p.K; ++i) {
      const unsigned long long key = sL[w][i];
      if (key <= th) break;
      list_insert(m, key, lane);
      th = __shfl_sync(0xffffffffu, m, p.K - 1);
    }
  emit_row(p, row, m, lane);
}

// The scan's lists of a row merged by one warp (up to 32 lists; eight rows per block).
constexpr int ROW_LISTS = 32;

__global__ void __launch_bounds__(FIN_WARPS * 32)
lmk_merge_rows_kernel(FinalParams p) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * FIN_WARPS + (threadIdx.x >> 5);
  pdl_trigger();
  pdl_wait();
  if (row >= p.R) return;
  const unsigned long long* src = p.keys + row * p.P + (long long)lane * p.K;
  emit_row(p, row, merge_heads(p.K, lane < p.lists, lane, [&](int i) { return src[i]; }), lane);
}

// Many lists per row (a long cache scanned by every SM), up to 160: one block per row.  All keys come to shared memory, 1,664 of them a trip, then one warp
// merges the lists, five a lane, by K warp-wide maxima of the heads' 32-bit scores: whose head it is notes the key and moves on.
// Equal scores move on together: more noted than rounds (looked at after two of them and at the end), and the warp starts again with the lowest id of each
// maximum, a second maximum a round; at once where scores are rounded to 16 bits, which are often equal.  (A vote in every round: K = 16 4 % more for distinct
// scores.  Lists an odd number of keys apart, in banks of their own: 3 % more, by the sums for it.)  1 x 5,000 of 768 per head, K = 16: distinct scores 10.0 us,
// rounded ones 11.6 (15.8 with the general way for equal scores, 10.7 when that had 256 threads), all equal 11.8 (16.3, 9.9).
// 128 threads and 8 bytes a key: up to a width of 768 and K = 15 a block finds its place beside one of the scan (192 KB + 15, 512 threads of up to 112
// registers) and is there when the scan ends.  With 256 threads it did not: 1 x 32,768 landmarks per head on all 148 SMs 20.4 us, on 128 of them 16.1.  Wider
// rows and longer lists leave it no place, and it starts when blocks of the scan have left; several of a launch then share an SM, so they must be
// short: ranked by counting as below, K = 32 took 30 us of 128 threads (20 of 256).  1 x 7,400 x 768, K = 16 / 32: 10.8 / 31.2 us, now 9.6 / 13.5;
// 1 x 266,400 per head, K = 32, x 768 97 (now 78), x 1,024 182 (101).
constexpr int WARP_LISTS = 160, MERGE_THREADS = 128, MERGE_LOADS = 13;

__global__ void __launch_bounds__(MERGE_THREADS)
lmk_warp_merge_kernel(FinalParams p) {
  extern __shared__ unsigned long long all[];                            // [lists][K]
  __shared__ unsigned long long best[MAXK];
  const int tid = threadIdx.x, K = p.K, keys = p.lists * K;
  const unsigned long long* src = p.keys + (long long)blockIdx.x * p.P;
  if (tid < MAXK) best[tid] = 0ull;
  pdl_trigger();
  pdl_wait();
  for (int i0 = tid; i0 < keys; i0 += MERGE_LOADS * MERGE_THREADS) {
    unsigned long long v[MERGE_LOADS];
#pragma unroll
    for (int i = 0; i < MERGE_LOADS; ++i) v[i] = i0 + i * MERGE_THREADS < keys ? src[i0 + i * MERGE_THREADS] : 0ull;
#pragma unroll
    for (int i = 0; i < MERGE_LOADS; ++i)
      if (i0 + i * MERGE_THREADS < keys) all[i0 + i * MERGE_THREADS] = v[i];
  }
  __syncthreads();
  if (tid >= 32) return;
  constexpr int MINE = WARP_LISTS / 32;
  unsigned h[MINE];
  int at[MINE];
  auto start = [&] {
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      at[i] = (tid + 32 * i) * K;
      h[i] = tid + 32 * i < p.lists ? (unsigned)(all[at[i]] >> 32) : 0u;
    }
  };
  auto highest = [&] {
    unsigned top = h[0];
#pragma unroll
    for (int i = 1; i < MINE; ++i) top = max(top, h[i]);
    return __reduce_max_sync(0xffffffffu, top);
  };
  auto take = [&](int i, int k) {                                        // the head of this lane's list i is the k-th best
    best[k] = all[at[i]];
    ++at[i];
    h[i] = at[i] < (tid + 32 * i + 1) * K ? (unsigned)(all[at[i]] >> 32) : 0u;
  };
  start();
  int k = 0, noted = p.score_round != 0;
  if (!p.score_round) {
    auto rounds = [&](int end) {
      for (; k < end; ++k) {
        const unsigned m = highest();
        if (m == 0u) return;
#pragma unroll
        for (int i = 0; i < MINE; ++i)
          if (h[i] == m) { take(i, k); ++noted; }
      }
    };
    rounds(min(K, 2));
    if (__reduce_add_sync(0xffffffffu, noted) == k) rounds(K);
  }
  if (__reduce_add_sync(0xffffffffu, noted) != k) {
    __syncwarp();
    start();
    unsigned low[MINE];                                                  // ~id of each head
#pragma unroll
    for (int i = 0; i < MINE; ++i) low[i] = h[i] ? (unsigned)all[at[i]] : 0u;
#pragma unroll 1
    for (k = 0; k < K; ++k) {
      const unsigned m = highest();
      if (m == 0u) break;
      unsigned mine = 0u;
#pragma unroll
      for (int i = 0; i < MINE; ++i) mine = max(mine, h[i] == m ? low[i] : 0u);
      if (mine != __reduce_max_sync(0xffffffffu, mine)) continue;
#pragma unroll
      for (int i = 0; i < MINE; ++i)
        if (low[i] == mine) { take(i, k); low[i] = h[i] ? (unsigned)all[at[i]] : 0u; }
    }
    if (tid >= k) best[tid] = 0ull;
  }
  __syncwarp();
  emit_row(p, blockIdx.x, tid < K ? best[tid] : 0ull, tid);
}

// More lists than that: no serial insertion either.  An entry e of a
// list can be among the K best only if fewer than K - e list heads are better than its own; so the heads are ranked by counting,
// the K best lists are lined up by rank, and their K (K + 1) / 2 possible entries are ranked by counting again.
// 296 lists, K = 8: 12.9 us of warp-serial insertions before.
constexpr int RANK_LISTS = 1024;

__global__ void __launch_bounds__(FIN_WARPS * 32)
lmk_rank_merge_kernel(FinalParams p) {
  __shared__ __align__(16) unsigned long long heads[RANK_LISTS];
  __shared__ int by_rank[MAXK];
  __shared__ unsigned long long cand[MAXK * (MAXK + 1) / 2 + 1], best[MAXK];
  const int tid = threadIdx.x, lists = p.lists, K = p.K;
  const int padded = (lists + 1) & ~1;
  const unsigned long long* src = p.keys + (long long)blockIdx.x * p.P;
  if (tid < MAXK) { by_rank[tid] = -1; best[tid] = 0ull; }
  pdl_trigger();
  pdl_wait();
  for (int i = tid; i < padded; i += FIN_WARPS * 32) heads[i] = i < lists ? src[(long long)i * K] : 0ull;
  __syncthreads();
  for (int i = tid; i < lists; i += FIN_WARPS * 32) {
    const unsigned long long mine = heads[i];
    if (mine == 0ull) continue;
    int rank = 0;
    for (int j = 0; j < padded; j += 2) {
      const ulonglong2 h = *reinterpret_cast<const ulonglong2*>(&heads[j]);
      rank += (h.x > mine) + (h.y > mine);
    }
    if (rank < K) by_rank[rank] = i;                      // keys are distinct: one list per rank
  }
  __syncthreads();
  // candidate (r, e), r + e < K, at position e of the list of rank r
  const int total = K * (K + 1) / 2;
  for (int i = tid; i < K * K; i += FIN_WARPS * 32) {
    const int r = i / K, e = i - r * K;
    if (r + e < K) cand[r * K - r * (r - 1) / 2 + e] = by_rank[r] >= 0 ? src[(long long)by_rank[r] * K + e] : 0ull;
  }
  __syncthreads();
  for (int i = tid; i < total; i += FIN_WARPS * 32) {
    const unsigned long long mine = cand[i];
    if (mine == 0ull) continue;
    int rank = 0;
    for (int j = 0; j < total; ++j) rank += cand[j] > mine;
    if (rank < K) best[rank] = mine;
  }
  __syncthreads();
  if (tid < 32) emit_row(p, blockIdx.x, tid < K ? best[tid] : 0ull, tid);
}

__global__ void __launch_bounds__(FIN_WARPS * 32)
lmk_finalize_kernel(FinalParams p) {
  __shared__ unsigned long long sL[FIN_WARPS][MAXK];
  finalize_row(p, blockIdx.x, p.keys + (long long)blockIdx.x * p.P, sL);
}

// ---------------------------------------------------------------------------------------------
// Candidate exchange between the GPUs of a chunk-range-sharded cache, fused with the merge.
//
// Every rank owns a MAILBOX in its own memory that the other ranks of the node have mapped
// (CUDA IPC).  One launch per rank and retrieval step: a block per query row
//   1. STORES this rank's K packed candidates of the row into its slot of every rank's mailbox
//      (plain stores through the peer mapping; over NVLink for the other GPUs),
//   2. raises its flag there (system-scope release after a system-scope fence),
//   3. waits -- for at most `wait_ns` -- until every rank's flag of this step stands in its OWN
//      mailbox (system-scope acquire loads of local memory),
//   4. merges the world x K candidates (same merge, same canonical order as on one GPU, so every
//      rank gets the identical result) and writes indices / scores / weights.
// No rank reads another GPU's memory and nothing is multicast: remote traffic is stores only.
// Steps are numbered by an epoch the kernel keeps in the mailbox header (one per row, advanced
// when the row's merge is done), so the launch can sit in a CUDA graph; two mailbox buffers
// alternate by epoch parity: a rank can be at most one step ahead of another (to finish step e
// it needs everybody's flag of step e), so a buffer is never overwritten while it is being read.
// When the wait expires the block raises GCA_STATUS_TIMEOUT, leaves the epoch where it was and
// returns: the context stays usable, and the host decides (PeerExchange.reset()).
//
// Mailbox layout (bytes): epoch[R_max] u32 | pad to 256 | 2 x { keys[R_max][world][MAXK] u64 |
// flags[R_max][world] u32 | pad to 256 }.
struct ExchangeParams {
  const unsigned long long* local_keys;     // (R, K)
  void* const* mailboxes;                   // device array of `world` pointers (this process's mappings)
  FinalParams fin;
  int32_t* status;
  int R, K, world, rank, r_max;
  unsigned long long wait_ns;
};

__host__ __device__ inline size_t exch_buf_bytes(int r_max, int world) {
  const size_t keys = (size_t)r_max * world * MAXK * 8, flags = (size_t)r_max * world * 4;
  return (keys + flags + 255) / 256 * 256;
}
__host__ __device__ inline size_t exch_hdr_bytes(int r_max) { return ((size_t)r_max * 4 + 255) / 256 * 256; }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__global__ void __launch_bounds__(FIN_WARPS * 32)
lmk_exchange_kernel(ExchangeParams p) {
  __shared__ unsigned long long sL[FIN_WARPS][MAXK];
  __shared__ int s_ok;
  const int row = blockIdx.x, tid = threadIdx.x;
  char* mine = static_cast<char*>(p.mailboxes[p.rank]);
  unsigned* epochs = reinterpret_cast<unsigned*>(mine);
  const unsigned e = *reinterpret_cast<volatile unsigned*>(epochs + row) + 1u;
  const size_t buf_off = exch_hdr_bytes(p.r_max) + (size_t)(e & 1u) * exch_buf_bytes(p.r_max, p.world);
  const size_t flags_off = buf_off + (size_t)p.r_max * p.world * MAXK * 8;
  // 1. my candidates into my slot of every rank's mailbox (thread = (destination rank, key); a
  //    slot is MAXK keys wide, the keys past K are written as "empty")
  if (tid < p.world * MAXK) {
    const int dst = tid / MAXK, i = tid - dst * MAXK;
    unsigned long long* slot = reinterpret_cast<unsigned long long*>(static_cast<char*>(p.mailboxes[dst]) + buf_off) +
                               ((size_t)row * p.world + p.rank) * MAXK;
    slot[i] = i < p.K ? p.local_keys[(size_t)row * p.K + i] : 0ull;
  }
  __threadfence_system();
  __syncthreads();
  // 2. my flag of this step in every rank's mailbox
  if (tid < p.world) {
    unsigned* flag = reinterpret_cast<unsigned*>(static_cast<char*>(p.mailboxes[tid]) + flags_off) + (size_t)row * p.world + p.rank;
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(e) : "memory");
  }
  // 3. bounded wait for every rank's flag in MY mailbox
  if (tid == 0) s_ok = 1;
  __syncthreads();
  if (tid < p.world) {
    const unsigned* flag = reinterpret_cast<const unsigned*>(mine + flags_off) + (size_t)row * p.world + tid;
    const unsigned long long t0 = global_ns();
    for (;;) {
      unsigned v;
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
      if (v == e) break;
      if (global_ns() - t0 > p.wait_ns) { s_ok = 0; break; }
      __nanosleep(200);
    }
  }
  __syncthreads();
  if (!s_ok) {
    if (tid == 0 && p.status) atomicOr(p.status, GCA_STATUS_TIMEOUT);
    return;
  }
  // 4. the row's candidates sit contiguously in my mailbox, MAXK per rank with empty keys (0) as
  //    filler: the merge takes them in place as P = world x MAXK candidates
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(mine + buf_off) + (size_t)row * p.world * MAXK;
  finalize_row(p.fin, row, src, sL);
  if (tid == 0) epochs[row] = e;
}

int pick_tq(const LmkTopkArgs& a) { return (a.head_dim > 0 || a.Cq < 4) ? 1 : 4; }

}  // namespace

// Two CTAs per SM when the query tile count alone does not fill the GPU.
int scan_splits(const LmkTopkArgs& a, int sms) {
  const int tq = pick_tq(a);
  const long long blocks = (long long)a.N * ((a.Cq + tq - 1) / tq);
  long long s = (2 * (long long)sms + blocks - 1) / blocks;
  const long long max_s = (a.E + 255) / 256;              // keep at least 256 rows per split
  if (s > max_s) s = max_s;
  if (s < 1) s = 1;
  return (int)s;
}

namespace {

// Landmark ranges of the streaming form: one block per SM at a time, so what counts is whole waves; a wave costs about as much
// again as reading 200 rows before and after its stream (32 rows x 4,096 landmarks: one wave of 4 ranges 36 us, two of 9 41; x 8,192
// 66 either way).
int most_stream_splits(const LmkTopkArgs& a, int sms) { return (int)std::min<long long>((a.E + SPLIT_ROWS - 1) / SPLIT_ROWS, 2 * sms); }
int stream_splits(const LmkTopkArgs& a, int sms) {
  const long long blocks = (long long)a.N * a.Cq;
  const int most = most_stream_splits(a, sms);
  int best = 1;
  long long best_cost = -1;
  for (int s = 1; s <= most; ++s) {
    const long long cost = (blocks * s + sms - 1) / sms * ((a.E + s - 1) / s + 200);
    if (best_cost < 0 || cost < best_cost) { best = s; best_cost = cost; }
  }
  // A block's warps take 64 rows at a time, 32 beyond a width of 768: of as many steps the fewest lists (4 x 8,192: 32 ranges of 256 rows 13.2 us, 37 of 222
  // 13.8).  Among a thousand rows a step is nothing, and all SMs read.  Nor are so many long lists given up that a warp merges them, which fetches entries as
  // it needs them, where the block had them all (4 x 2,442 to 4,810 landmarks, K = 16: 5 to 10 % more; K = 8: 4 x 3,700 of 1,024 per head 8 % less).  2,500
  // sizes of 66 to 1,000 rows a block, widths of 256 to 1,024, K = 8 and 16: 1.4 % less than without steps on average, at most 4 % more in 99 of 100.
  const int step = STREAM_WARPS * (a.D > 768 ? ROWS_AT_ONCE<4> : ROWS_AT_ONCE<3>), rows = (a.E + best - 1) / best;
  if (rows > 0 && rows < 1024) {
    const int taken = (rows + step - 1) / step * step, fewest = (a.E + taken - 1) / taken;
    if (a.K <= 8 || best <= ROW_LISTS || fewest > ROW_LISTS) best = fewest;
  }
  return best;
}

int choose_splits(const LmkTopkArgs& a, int sms) {
  return a.splits > 0 ? a.splits : pick_tq(a) == 1 ? stream_splits(a, sms) : scan_splits(a, sms);
}

// A row's blocks are a cluster that merges for itself where they are at most eight anyway and all clusters find their SMs, in one group of
// them each: 256 landmarks x 1 row 6.9 us either way (the merge kernel is on its way before the scan ends) but one launch less on
// the host, calls in a row 9.1 -> 7.3 us; 64 landmarks 6.6 -> 5.7 us.  A cluster of eight in place of more blocks costs more than it saves
// (1,000 landmarks: 16 blocks and a merge 6.7 us, a cluster 9.2).
bool fused(const LmkTopkArgs& a, int splits, int sms) {
  const int slack = splits == 1 ? 0 : splits < 5 ? 1 : splits;
  return splits <= 8 && (long long)a.N * a.Cq * splits * (16 + slack) <= 16ll * sms;
}

template <int NP, bool PER_HEAD, bool FUSED>
int launch_stream(const ScanParams& sp, const FinalParams& fp, dim3 grid, cudaStream_t stream) {
  constexpr int smem = STREAM_WARPS * RING_ROWS<NP> * NP * 512;
  auto kernel = lmk_stream_kernel<NP, PER_HEAD, FUSED>;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(STREAM_WARPS * 32); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = grid.x; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = FUSED && grid.x > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, sp, fp);
}

template <int NP>
int launch_scan(const ScanParams& sp, const FinalParams& fp, int tq, bool per_head, bool fused, cudaStream_t stream) {
  const dim3 grid((unsigned)sp.splits, (unsigned)((sp.Cq + tq - 1) / tq), (unsigned)sp.N);
  if (per_head) return fused ? launch_stream<NP, true, true>(sp, fp, grid, stream) : launch_stream<NP, true, false>(sp, fp, grid, stream);
  if (tq == 1) return fused ? launch_stream<NP, false, true>(sp, fp, grid, stream) : launch_stream<NP, false, false>(sp, fp, grid, stream);
  lmk_scan_kernel<NP, 4><<<grid, SCAN_WARPS * 32, 0, stream>>>(sp);
  return (int)cudaGetLastError();
}

}  // namespace

size_t lmk_topk_rows(const LmkTopkArgs& a) {
  const int H = a.head_dim > 0 ? a.D / a.head_dim : 1;
  return (size_t)a.N * a.Cq * H;
}

// sms = 0: what any device of up to 256 SMs needs.  Screening and the row scan take more lists the more SMs there are; the streaming
// form does not (5 rows x 262,144: 59 lists for 148 SMs, 51 for 256), so there the most it tries counts.
size_t lmk_topk_workspace_bytes_impl(const LmkTopkArgs& a, int sms) {
  const int assumed = sms > 0 ? sms : 256;
  if (lmk_screen_applies(a)) return lmk_screen_workspace_bytes(a, assumed);
  const int splits = sms == 0 && a.splits == 0 && pick_tq(a) == 1 ? std::max(1, most_stream_splits(a, assumed)) : choose_splits(a, assumed);
  return align_up(lmk_topk_rows(a) * (size_t)splits * a.K * sizeof(unsigned long long), 256);
}

// Scan + merge on caller-provided scratch.  `scratch` must hold
// lmk_topk_workspace_bytes_impl(a, sms) bytes.
int launch_lmk_score_topk(const LmkTopkArgs& a, void* scratch, int sms, cudaStream_t stream, int32_t* kept_indices, float* kept_weights) {
  const size_t rows = lmk_topk_rows(a);
  if (rows == 0) return 0;
  const bool per_head = a.head_dim > 0;
  const float scale = (float)(1.0 / sqrt((double)(per_head ? a.head_dim : a.D)));
  FinalParams fp;
  fp.keys = (unsigned long long*)scratch; fp.out_keys = (unsigned long long*)a.out_keys; fp.out_indices = a.out_indices;
  fp.out_scores = a.out_scores; fp.out_weights = a.out_weights; fp.out_nvalid = a.out_nvalid;
  fp.kept_indices = kept_indices; fp.kept_weights = kept_weights;
  fp.lq = (const __nv_bfloat16*)a.lmk_q; fp.lk = (const __nv_bfloat16*)a.lmk_k;
  fp.qbs = a.q_batch_stride; fp.qrs = a.q_row_stride; fp.kbs = a.k_batch_stride; fp.krs = a.k_row_stride; fp.e_base = a.e_base;
  fp.Cq = a.Cq; fp.D = a.D; fp.score_round = a.score_round; fp.scale = scale;
  fp.R = (int)rows; fp.P = 0; fp.K = a.K; fp.lists = 0;
  if (lmk_screen_applies(a)) return launch_lmk_screen(a, scratch, sms, fp, stream);
  const int tq = pick_tq(a), splits = choose_splits(a, sms);
  const bool cluster = tq == 1 && fused(a, splits, sms);
  if (a.noise == nullptr || per_head) fp.lq = nullptr;          // the keys hold the noise-free scores
  fp.P = splits * a.K; fp.lists = splits;
  ScanParams sp;
  sp.lq = (const __nv_bfloat16*)a.lmk_q; sp.lk = fp.lk; sp.noise = a.noise;
  sp.part = (unsigned long long*)scratch;
  sp.qbs = a.q_batch_stride; sp.qrs = a.q_row_stride; sp.kbs = a.k_batch_stride; sp.krs = a.k_row_stride;
  sp.q_pos0 = a.q_pos0; sp.e_base = a.e_base;
  sp.N = a.N; sp.Cq = a.Cq; sp.E = a.E; sp.D = a.D; sp.K = a.K; sp.H = per_head ? a.D / a.head_dim : 1;
  sp.splits = splits; sp.e_per_split = (a.E + splits - 1) / splits;
  sp.score_round = a.score_round; sp.scale = scale;
  int rc;
  switch ((a.D + 255) / 256) {
    case 1: rc = launch_scan<1>(sp, fp, tq, per_head, cluster, stream); break;
    case 2: rc = launch_scan<2>(sp, fp, tq, per_head, cluster, stream); break;
    case 3: rc = launch_scan<3>(sp, fp, tq, per_head, cluster, stream); break;
    case 4: rc = launch_scan<4>(sp, fp, tq, per_head, cluster, stream); break;
    default: rc = GCA_ERR_SHAPE;
  }
  if (rc) return rc;
  if (cluster) return 0;
  // a warp per row up to 32 lists, a block per row beyond
  if (splits <= ROW_LISTS)
    return (int)launch_dependent(lmk_merge_rows_kernel, dim3((unsigned)((rows + FIN_WARPS - 1) / FIN_WARPS)), dim3(FIN_WARPS * 32), 0, stream, fp);
  if (splits <= WARP_LISTS)
    return (int)launch_dependent(lmk_warp_merge_kernel, dim3((unsigned)rows), dim3(MERGE_THREADS), (size_t)splits * a.K * sizeof(unsigned long long), stream, fp);
  if (splits <= RANK_LISTS) return (int)launch_dependent(lmk_rank_merge_kernel, dim3((unsigned)rows), dim3(FIN_WARPS * 32), 0, stream, fp);
  lmk_finalize_kernel<<<(unsigned)rows, FIN_WARPS * 32, 0, stream>>>(fp);
  return (int)cudaGetLastError();
}

int launch_lmk_merge(const LmkMergeArgs& a, cudaStream_t stream) {
  if (a.R == 0) return 0;
  FinalParams fp;
  fp.keys = (const unsigned long long*)a.keys; fp.out_keys = (unsigned long long*)a.out_keys; fp.out_indices = a.out_indices; fp.out_scores = a.out_scores;
  fp.out_weights = a.out_weights; fp.out_nvalid = a.out_nvalid;
  fp.lq = nullptr; fp.lk = nullptr; fp.qbs = fp.qrs = fp.kbs = fp.krs = fp.e_base = 0;
  fp.Cq = 1; fp.D = 0; fp.score_round = 0; fp.scale = 1.f;
  fp.R = a.R; fp.P = a.P; fp.K = a.K; fp.lists = 0;
  lmk_finalize_kernel<<<(unsigned)a.R, FIN_WARPS * 32, 0, stream>>>(fp);
  return (int)cudaGetLastError();
}

}  // namespace gca

// ---------------------------------------------------------------------------------------------
// lmk_score_topk_static: the same scan + finalize, for callers that cannot hand us scratch.
//
// Who needs this: a host that must not (or cannot) allocate device memory around the call --
// for example a serving process that gave all of HBM to its own pools at start-up, a plugin
// living inside another framework whose allocator it may not touch, or a latency-critical loop
// where an allocator call (and the device-wide synchronisation it can imply) is not acceptable.
// Such a caller still passes its inputs and outputs, but the per-block candidate lists go into
// a fixed array that lives in the library image.
//
// The array is file-scope device memory: every GPU that loads this library carries it
// (LMK_STATIC_SCRATCH_BYTES = 1 MiB) until the process exits.  In host code its name is only a
// stand-in for the symbol, not a device address, so the address is looked up with
// cudaGetSymbolAddress -- once per device, with that device current (the device that holds the
// landmark cache, made current for the call), on the first call made for that device -- and only
// that looked-up pointer is handed to the kernels.  Because of that
// look-up, make the first call on each device before starting any stream capture.
//
// All calls on one GPU share the array.  It keeps whatever the previous call left in it; that
// is harmless here because a call writes every (row, split) list it later reads, so nothing
// needs to start at zero.  Two calls that overlap on the same GPU (different streams, or
// different host threads) would overwrite each other's lists: serialise them.
// ---------------------------------------------------------------------------------------------
#include <cstring>
#include <mutex>

namespace gca {
namespace {

static __device__ __align__(256) unsigned long long g_lmk_static_scratch[LMK_STATIC_SCRATCH_BYTES / 8];

constexpr int MAX_DEVICES = 64;
std::mutex g_static_mu;
void* g_static_ptr[MAX_DEVICES] = {};

// Device address of the static scratch on device `dev`, which must be current (resolved once per device).
int static_scratch_ptr(int dev, void** out) {
  if (dev < 0 || dev >= MAX_DEVICES) return GCA_ERR_TOO_LARGE;
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    GCA_CUDA_CHECK(cudaGetSymbolAddress(&p, g_lmk_static_scratch));
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return 0;
}

}  // namespace
}  // namespace gca

extern "C" int lmk_score_topk_static(const LmkTopkArgs* a, void* stream) {
  // same argument rules as lmk_score_topk; `workspace` / `workspace_bytes` are ignored
  int rc = gca::check_topk(a);
  if (rc) return rc;
  if (a->N == 0 || a->Cq == 0) return 0;
  gca::DeviceScope scope(a->lmk_k);        // the array of the GPU that holds the landmarks
  if (scope.rc) return scope.rc;
  const int sms = gca::sm_count(scope.dev);
  // rows x splits x K candidate keys of 8 bytes must fit the built-in array: the row scan needs the fewest lists
  LmkTopkArgs b = *a;
  if (b.splits == 0) b.splits = gca::scan_splits(b, sms);
  a = &b;
  if (gca::lmk_topk_workspace_bytes_impl(*a, sms) > (size_t)LMK_STATIC_SCRATCH_BYTES) return GCA_ERR_STATIC_SCRATCH;
  void* scratch = nullptr;
  rc = gca::static_scratch_ptr(scope.dev, &scratch);
  if (rc) return rc;
  return gca::launch_lmk_score_topk(*a, scratch, sms, (cudaStream_t)stream, nullptr, nullptr);
}

// ---------------------------------------------------------------------------------------------
// Host side of the candidate exchange: mailbox set-up (CUDA IPC) and the launch.
// ---------------------------------------------------------------------------------------------
extern "C" size_t lmk_exchange_mailbox_bytes(int r_max, int world) {
  if (r_max < 1 || world < 1) return 0;
  return gca::exch_hdr_bytes(r_max) + 2 * gca::exch_buf_bytes(r_max, world);
}

extern "C" int lmk_exchange_mailbox_create(int r_max, int world, void** mailbox, void* ipc_handle64) {
  if (!mailbox || !ipc_handle64) return GCA_ERR_NULL;
  if (r_max < 1 || world < 1 || world > 8) return GCA_ERR_SHAPE;
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the handle is exchanged as 64 bytes");
  const size_t bytes = lmk_exchange_mailbox_bytes(r_max, world);
  void* p = nullptr;
  GCA_CUDA_CHECK(cudaMalloc(&p, bytes));
  cudaError_t e = cudaMemset(p, 0, bytes);
  if (e == cudaSuccess) e = cudaIpcGetMemHandle(static_cast<cudaIpcMemHandle_t*>(ipc_handle64), p);
  if (e != cudaSuccess) { cudaFree(p); return (int)e; }
  *mailbox = p;
  return 0;
}

extern "C" int lmk_exchange_mailbox_open(const void* ipc_handle64, void** peer_ptr) {
  if (!ipc_handle64 || !peer_ptr) return GCA_ERR_NULL;
  cudaIpcMemHandle_t h;
  memcpy(&h, ipc_handle64, sizeof(h));
  GCA_CUDA_CHECK(cudaIpcOpenMemHandle(peer_ptr, h, cudaIpcMemLazyEnablePeerAccess));
  return 0;
}

extern "C" int lmk_exchange_mailbox_close(void* peer_ptr) {
  if (!peer_ptr) return GCA_ERR_NULL;
  GCA_CUDA_CHECK(cudaIpcCloseMemHandle(peer_ptr));
  return 0;
}

extern "C" int lmk_exchange_mailbox_destroy(void* mailbox) {
  if (!mailbox) return GCA_ERR_NULL;
  GCA_CUDA_CHECK(cudaFree(mailbox));
  return 0;
}

extern "C" int lmk_exchange_mailbox_reset(void* mailbox, int r_max, int world, void* stream) {
  if (!mailbox) return GCA_ERR_NULL;
  GCA_CUDA_CHECK(cudaMemsetAsync(mailbox, 0, lmk_exchange_mailbox_bytes(r_max, world), (cudaStream_t)stream));
  return 0;
}

extern "C" int lmk_topk_exchange(const LmkExchangeArgs* a, void* stream) {
  if (!a) return GCA_ERR_NULL;
  if (!a->local_keys || !a->mailboxes || !a->out_keys) return GCA_ERR_NULL;
  if (a->world < 1 || a->world > 8 || a->rank < 0 || a->rank >= a->world) return GCA_ERR_SHAPE;
  if (a->R < 0 || a->R > a->R_max || a->K < 1 || a->K > gca::MAXK) return GCA_ERR_SHAPE;
  if (a->R == 0) return 0;
  gca::DeviceScope scope(a->local_keys);
  if (scope.rc) return scope.rc;
  gca::ExchangeParams p;
  p.local_keys = reinterpret_cast<const unsigned long long*>(a->local_keys);
  p.mailboxes = a->mailboxes;
  p.status = a->status;
  p.R = a->R; p.K = a->K; p.world = a->world; p.rank = a->rank; p.r_max = a->R_max;
  p.wait_ns = (unsigned long long)(a->wait_ms > 0 ? a->wait_ms : 1000) * 1000000ull;
  gca::FinalParams& fp = p.fin;
  fp.keys = nullptr; fp.out_keys = reinterpret_cast<unsigned long long*>(a->out_keys); fp.out_indices = a->out_indices;
  fp.out_scores = a->out_scores; fp.out_weights = a->out_weights; fp.out_nvalid = a->out_nvalid;
  fp.lq = nullptr; fp.lk = nullptr; fp.qbs = fp.qrs = fp.kbs = fp.krs = fp.e_base = 0;
  fp.Cq = 1; fp.D = 0; fp.score_round = 0; fp.scale = 1.f;
  fp.R = a->R; fp.P = a->world * gca::MAXK; fp.K = a->K; fp.lists = 0;
  gca::lmk_exchange_kernel<<<(unsigned)a->R, gca::FIN_WARPS * 32, 0, (cudaStream_t)stream>>>(p);
  return (int)cudaGetLastError();
}
