// Landmark top-k for many query rows per sequence (a training step, a prefill) on the tensor cores, with the bits of
// the row scan.
//
// Scoring every (row, landmark) pair is a matrix product, but the selection is defined on float32 sums in ONE fixed order
// (lmk_topk.cu), which a tensor core does not follow.  So the product only SCREENS: it gives every score to within a bound, a
// row keeps its KC = K + 4 best approximate scores per range of landmarks, and the merge computes the exact score of
// those that can still be among the K best -- K of them, rarely one more -- in the scan's own order.
//
//   |approximate - exact| <= 2^-15 |q| |k| / sqrt(D) =: eps.   Either sum of exact bf16 products is off by at most a few dozen
//   roundings of 2^-24 of sum |q_i k_i| <= |q| |k|; tensor cores align and truncate at 2^-22 or better per addition, 48 of
//   them for D = 768.  The bound is ~8e-4 of the spread of the scores of one row, so it costs next to nothing.
//   With T the K-th best approximate score of the row, whatever lies below T - 2 eps cannot win.  A range whose KC
//   entries are all above that line may hide more (copies of one landmark): that row is scanned exactly by its block.
//
// Screening: one CTA per (128 rows, range of landmarks), tiles of 64 landmarks; warp 16 issues the TMA copies of a 7-stage ring
// (128 x 64 of q, 64 x 64 of the landmarks), warp 17 the 128 x 64 x 16 MMAs.  Of 16 worker warps the first six add up the squared norms
// from the same stages while they pass; then a thread takes 16 scores of one row from tensor memory and sorts them in its
// registers, and the four runs of a row are merged in two steps through shared memory, the last with the row's list so far.
// Every wait is bounded; when one runs out the error bound of the block's rows is written as infinite, which sends them through the
// exact scan.  What bounds it is latency (12 K steps, one selection round after another): 8 x 260 rows x 260 landmarks x 768
// take 15 us of screening and 14 of settling (each by itself, cold), 31 us as a call; the row scan and its merge 142.
#include <algorithm>

#include "lmk_common.cuh"
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

namespace gca {

namespace {

using namespace sm100;

constexpr int BM = 128, BN = 64, BK = 64, STAGES = 7;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int WORKERS = 16, THREADS = (WORKERS + 2) * 32, NORM_WARPS = (BM + BN) / 32;
constexpr int COLS = 16;                          // score columns per worker thread
constexpr int OFF_X1 = STAGES * STAGE_BYTES;      // [2 tiles][2 pairs of column groups][COLS][BM] keys
constexpr int OFF_X2 = OFF_X1 + 4 * COLS * BM * 4, OFF_NORM = OFF_X2 + 32 * BM * 4, OFF_BAR = OFF_NORM + 2 * (BM + BN) * 4;
static_assert(OFF_BAR + 256 + 1024 <= 227 * 1024, "shared memory");
constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
constexpr int EXTRA = 4, MAX_LISTS = 32;
constexpr float BOUND = 1.0f / 32768.0f;
enum Bar { FULL = 0, EMPTY = FULL + STAGES, ACC_FULL = EMPTY + STAGES, ACC_EMPTY, NUM_BARS };
constexpr uint32_t IDESC = umma_idesc_bf16(BM, BN, 0, 0);

struct ScreenParams {
  CUtensorMap tm_q, tm_k;
  const float* noise;
  unsigned long long* part;      // (rows, lists, KC) approximate keys, descending
  float* eps;                    // (rows, lists)
  long long q_pos0, e_base;
  int Cq, E, D, KC, lists, tiles_per_list;
  int noise_vec;                 // the noise can be read as float4
  float scale;
};

// Sorting networks on a thread's own registers, descending; every index is a constant.
template <class T>
__device__ __forceinline__ void order(T& hi, T& lo) {
  const T a = hi, b = lo;
  hi = a > b ? a : b;
  lo = a > b ? b : a;
}
template <int LO, int N, int R, class T>
__device__ __forceinline__ void odd_even_merge(T* v) {
  if constexpr (2 * R < N) {
    odd_even_merge<LO, N, 2 * R>(v);
    odd_even_merge<LO + R, N, 2 * R>(v);
#pragma unroll
    for (int i = LO + R; i + R < LO + N; i += 2 * R) order(v[i], v[i + R]);
  } else {
    order(v[LO], v[LO + R]);
  }
}
template <int LO, int N, class T>
__device__ __forceinline__ void odd_even_sort(T* v) {      // Batcher's odd-even merge sort: 63 exchanges for 16 keys
  if constexpr (N > 1) {
    odd_even_sort<LO, N / 2>(v);
    odd_even_sort<LO + N / 2, N / 2>(v);
    odd_even_merge<LO, N, 1>(v);
  }
}
template <int N, class T>
__device__ __forceinline__ void bitonic_merge(T* v) {      // v: a descending run followed by an ascending one
#pragma unroll
  for (int d = N / 2; d > 0; d /= 2)
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (!(i & d)) order(v[i], v[i + d]);
}

template <int LEN>                // entries a thread keeps: KC <= LEN
__global__ void __launch_bounds__(THREADS, 1)
lmk_screen_kernel(const __grid_constant__ ScreenParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned* x1 = reinterpret_cast<unsigned*>(smem + OFF_X1);
  unsigned* x2 = reinterpret_cast<unsigned*>(smem + OFF_X2);
  float* norms = reinterpret_cast<float*>(smem + OFF_NORM);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + NUM_BARS + 1);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int list = blockIdx.x, t0 = blockIdx.y * BM, n = blockIdx.z;
  const int rows = min(BM, p.Cq - t0), ksteps = p.D / BK;
  // tiles of this list that some row of the block can see
  const int tiles_all = (p.E + BN - 1) / BN, first = list * p.tiles_per_list;
  const long long seen = p.q_pos0 + t0 + rows - 1 - p.e_base;             // landmarks visible to the last row
  const int last = (int)min((long long)min(tiles_all, first + p.tiles_per_list), seen <= 0 ? 0ll : (seen + BN - 1) / BN);
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&bars[FULL + i], 1); mbar_init(&bars[EMPTY + i], 1 + NORM_WARPS); }
    mbar_init(&bars[ACC_FULL], 1);
    mbar_init(&bars[ACC_EMPTY], WORKERS);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == WORKERS + 1) { tmem_alloc(tmem_slot, 64); tmem_relinquish(); }
  if (warp == WORKERS && lane == 0) { tma_prefetch_desc(&p.tm_q); tma_prefetch_desc(&p.tm_k); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  pdl_wait();
  const uint32_t tmem = *tmem_slot;

  if (warp == WORKERS) {
    uint32_t it = 0;
    bool ok = true;
    for (int t = first; t < last && ok; ++t)
      for (int ks = 0; ks < ksteps; ++ks, ++it) {
        const uint32_t st = it % STAGES;
        ok = mbar_wait_warp(&bars[EMPTY + st], ((it / STAGES) & 1) ^ 1, abort_flag, lane);
        if (!ok) break;
        mbar_expect_tx_elect(&bars[FULL + st], STAGE_BYTES);
        tma_load_3d_elect(smem + st * STAGE_BYTES, &p.tm_q, &bars[FULL + st], ks * BK, t0, n);
        tma_load_3d_elect(smem + st * STAGE_BYTES + A_BYTES, &p.tm_k, &bars[FULL + st], ks * BK, t * BN, n);
      }
    if (*abort_flag)          // nothing may land in shared memory after the block has gone
      for (uint32_t back = 0; back < (uint32_t)STAGES && back < it; ++back) {
        const uint32_t g = it - 1 - back;
        for (int i = 0; i < (1 << 20); ++i)
          if (mbar_try_wait(&bars[FULL + g % STAGES], (g / STAGES) & 1)) break;
      }
  } else if (warp == WORKERS + 1) {
    uint32_t it = 0, tile = 0;
    bool ok = true;
    for (int t = first; t < last && ok; ++t, ++tile) {
      ok = mbar_wait_warp(&bars[ACC_EMPTY], (tile & 1) ^ 1, abort_flag, lane);
      for (int ks = 0; ks < ksteps && ok; ++ks, ++it) {
        const uint32_t st = it % STAGES;
        ok = mbar_wait_warp(&bars[FULL + st], (it / STAGES) & 1, abort_flag, lane);
        if (!ok) break;
        tc_fence_after();
        const uint64_t da = umma_desc_sw128(smem_u32(smem + st * STAGE_BYTES)), db = umma_desc_sw128(smem_u32(smem + st * STAGE_BYTES + A_BYTES));
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) umma_bf16_ss_elect(tmem, da + kk * 2, db + kk * 2, IDESC, (uint32_t)(ks > 0 || kk > 0));
        umma_commit_elect(&bars[EMPTY + st]);
      }
      if (ok) umma_commit_elect(&bars[ACC_FULL]);
    }
  } else {
    bool ok = true;
    uint32_t it = 0, tile = 0;
    // thread: one row of the tile, COLS of its columns
    const int quad = warp & 3, group = warp >> 2, r = quad * 32 + lane, row = t0 + r, c0 = group * COLS;
    const bool live = r < rows;
    const long long grow = (long long)n * p.Cq + row;
    float eps_max = 0.f;                                     // of the row (group 0)
    unsigned long long* dst = p.part + (grow * p.lists + list) * p.KC;
    for (int t = first; t < last && ok; ++t, ++tile) {
      float* norm = norms + (tile & 1) * (BM + BN);
      if (warp < NORM_WARPS) {
        float ss[4] = {0.f, 0.f, 0.f, 0.f};
        for (int ks = 0; ks < ksteps && ok; ++ks, ++it) {
          const uint32_t st = it % STAGES;
          ok = mbar_wait_warp(&bars[FULL + st], (it / STAGES) & 1, abort_flag, lane);
          if (!ok) break;
          const uint8_t* src = smem + st * STAGE_BYTES + threadIdx.x * 128;        // A rows, then B rows right behind them
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            float f[8];
            unpack8(*reinterpret_cast<const uint4*>(src + ((c ^ (lane & 7)) << 4)), f);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss[i & 3] = fmaf(f[i], f[i], ss[i & 3]);
          }
          mbar_arrive_warp(&bars[EMPTY + st], lane);
        }
        norm[threadIdx.x] = (ss[0] + ss[1]) + (ss[2] + ss[3]);
      }
      // the row's noise while the products are being formed; columns the row cannot see become key 0
      const long long e0 = (long long)t * BN + c0;
      const int see = live ? (int)max(0ll, min((long long)COLS, min((long long)p.E - e0, p.q_pos0 + row - p.e_base - e0))) : 0;
      float add[COLS];
#pragma unroll
      for (int i = 0; i < COLS; ++i) add[i] = 0.f;
      if (p.noise) {
        const float* src = p.noise + grow * p.E + e0;
        if (p.noise_vec) {
#pragma unroll
          for (int i = 0; i < COLS; i += 4)
            if (i < see) {                                   // whole groups of four lie inside the row or outside
              const float4 v = *reinterpret_cast<const float4*>(src + i);
              add[i] = v.x; add[i + 1] = v.y; add[i + 2] = v.z; add[i + 3] = v.w;
            }
        } else {
#pragma unroll
          for (int i = 0; i < COLS; ++i)
            if (i < see) add[i] = src[i];
        }
      }
      if (ok) ok = mbar_wait_warp(&bars[ACC_FULL], tile & 1, abort_flag, lane);
      unsigned key[LEN];
      if (ok) {
        tc_fence_after();
        uint32_t v[COLS];
        tmem_ld_32x32b_x16(tmem + ((uint32_t)(quad * 32) << 16) + c0, v);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive_warp(&bars[ACC_EMPTY], lane);
        // key: the score without its last six bits, then the column, lower columns above; never equal inside a tile
#pragma unroll
        for (int i = 0; i < COLS; ++i)
          key[i] = i < see ? (orderable(__uint_as_float(v[i]) * p.scale + add[i]) & ~63u) | (unsigned)(BN - 1 - c0 - i) : 0u;
        odd_even_sort<0, COLS>(key);
        if (group & 1) {
#pragma unroll
          for (int i = 0; i < COLS; ++i) x1[(((tile & 1) * 2 + (group >> 1)) * COLS + i) * BM + r] = key[i];
        }
      }
      // one decision for all workers: whether any of them gave up
      int failed = !ok || *abort_flag;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\t"
          "setp.ne.s32 q, %0, 0;\n\t"
          "barrier.cta.red.or.pred p, 1, %1, q;\n\t"
          "selp.s32 %0, 1, 0, p;\n\t}"
          : "+r"(failed)
          : "r"(WORKERS * 32)
          : "memory");
      if (failed) { ok = false; break; }
      if (group & 1) continue;
      // two sorted runs of 16 -> the LEN best, sorted
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        const unsigned o = x1[(((tile & 1) * 2 + (group >> 1)) * COLS + COLS - 1 - i) * BM + r];
        if (LEN == COLS) key[i] = max(key[i], o);
        else key[LEN - COLS + i] = o;
      }
      bitonic_merge<LEN>(key);
      if (group == 2) {
#pragma unroll
        for (int i = 0; i < LEN; ++i) x2[i * BM + r] = key[i];
      }
      asm volatile("bar.sync 2, %0;" ::"r"(WORKERS * 16) : "memory");
      if (group == 2) continue;
#pragma unroll
      for (int i = 0; i < LEN; ++i) key[i] = max(key[i], x2[(LEN - 1 - i) * BM + r]);
      bitonic_merge<LEN>(key);
      // squared norms are never negative: as whole numbers they are in order, and a NaN is above them all
      const float kmax = __uint_as_float(__reduce_max_sync(0xffffffffu, max(__float_as_uint(norm[BM + lane]), __float_as_uint(norm[BM + 32 + lane]))));
      if (live) {
        const float bound = BOUND * p.scale * sqrtf(norm[r]) * sqrtf(kmax) * 1.001f;
        eps_max = fmaxf(eps_max, bound < 1e30f ? bound : INFINITY);      // NaN too: nothing is known about the tile, the row is scanned
        auto entry = [&](unsigned k) {
          return k ? (unsigned long long)(k & ~63u) << 32 | (0xffffffffu - (unsigned)(p.e_base + t * BN + (BN - 1) - (int)(k & 63u))) : 0ull;
        };
        if (t == first) {
#pragma unroll
          for (int i = 0; i < LEN; ++i)
            if (i < p.KC) dst[i] = entry(key[i]);
        } else {                                                 // with the list so far (this thread wrote it)
          unsigned long long run[LEN];
#pragma unroll
          for (int i = 0; i < LEN; ++i) {
            const unsigned long long o = i < p.KC ? dst[i] : 0ull, e = entry(key[LEN - 1 - i]);
            run[i] = o > e ? o : e;
          }
          bitonic_merge<LEN>(run);
#pragma unroll
          for (int i = 0; i < LEN; ++i)
            if (i < p.KC) dst[i] = run[i];
        }
      }
      __syncwarp();
    }
    if (group == 0 && live) {
      p.eps[grow * p.lists + list] = ok ? eps_max : INFINITY;      // a wait ran out: the merge scans the row itself
      if (last <= first)
        for (int i = 0; i < p.KC; ++i) dst[i] = 0ull;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WORKERS + 1) tmem_dealloc(tmem, 64);
}

struct SettleParams {
  FinalParams fin;
  const unsigned long long* part;
  const float* eps;
  const float* noise;
  long long q_pos0;
  int KC, lists, E;
  int rows;                      // of a block, one per warp
};

constexpr int SETTLE_WARPS = 8;

// Four landmark rows against the query row a warp holds: the scan's own sums, every lane gets them.
template <int NP>
__device__ __forceinline__ void exact_dot4(float s[4], const uint4 (&qv)[NP], const uint4 (&kv)[4][NP]) {
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    float acc = 0.f;
#pragma unroll
    for (int pp = 0; pp < NP; ++pp) {                      // absent pieces add 0 * 0: the sums never are -0
      float af[8], bf[8];
      unpack8(qv[pp], af);
      unpack8(kv[x][pp], bf);
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) acc = fmaf(af[jj], bf[jj], acc);
    }
#pragma unroll
    for (int of = 16; of > 0; of >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, of);
    s[x] = acc;
  }
}
template <int NP>
__device__ __forceinline__ void load_row(uint4 (&v)[NP], const __nv_bfloat16* src, int pieces, int lane) {
#pragma unroll
  for (int pp = 0; pp < NP; ++pp) v[pp] = lane + 32 * pp < pieces ? *reinterpret_cast<const uint4*>(src + (lane + 32 * pp) * 8) : make_uint4(0, 0, 0, 0);
}

// One warp: the candidates of a row that can win get their exact scores and are put in order.  False: the lists may hide a winner.
template <int NP>
__device__ __forceinline__ bool settle_row(const SettleParams& p, long long row, unsigned long long* won_key, float* won_score, int lane) {
  const FinalParams& f = p.fin;
  const long long n = row / f.Cq, r = row % f.Cq;
  const __nv_bfloat16* kb = f.lk + n * f.kbs;
  const int pieces = f.D >> 3;
  const unsigned long long* src = p.part + (row * p.lists + lane) * p.KC;
  const bool have = lane < p.lists;
  unsigned long long head = have ? src[0] : 0ull, next = have ? src[1] : 0ull, c0 = 0ull, c1 = 0ull;
  const unsigned eb = __reduce_max_sync(0xffffffffu, have ? __float_as_uint(p.eps[row * p.lists + lane]) : 0u);
  const float eps = __uint_as_float(eb);
  if (!(eps < 1e30f)) return false;
  float line = -INFINITY;
  int at = 1, count = 0;
  for (;;) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(head >> 32));
    if (hi == 0u) break;
    const float s = from_orderable(hi);
    if (count >= f.K && s < line) break;
    if (count == 64 || !(fabsf(s) < 1e30f)) return false;
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(head >> 32) == hi ? (unsigned)head : 0u);
    const unsigned long long best = ((unsigned long long)hi << 32) | lo;
    if (lane == (count & 31)) { if (count < 32) c0 = best; else c1 = best; }
    ++count;
    if (count == f.K) line = s - 2.001f * eps - fabsf(s) * 8.2e-6f;         // 2^-17: the bits a key leaves out; roundings of scale and noise
    bool spent = false;
    if (head == best) { head = next; ++at; next = at < p.KC ? src[at] : 0ull; spent = at > p.KC; }
    if (__any_sync(0xffffffffu, spent)) return false;                        // a full list used up: it may hide more
  }
  // exact scores; the rows of four candidates are requested together
  unsigned long long k0 = 0ull, k1 = 0ull;
  float s0 = 0.f, s1 = 0.f;
  uint4 qv[NP];
  load_row<NP>(qv, f.lq + n * f.qbs + r * f.qrs, pieces, lane);
  for (int i0 = 0; i0 < count; i0 += 4) {
    uint4 kv[4][NP];
    unsigned id[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int i = min(i0 + x, count - 1);
      id[x] = 0xffffffffu - (unsigned)__shfl_sync(0xffffffffu, i < 32 ? c0 : c1, i & 31);
      load_row<NP>(kv[x], kb + ((long long)id[x] - f.e_base) * f.krs, pieces, lane);
    }
    float acc[4];
    exact_dot4<NP>(acc, qv, kv);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float s = acc[x] * f.scale;
      const int i = i0 + x;
      if (i < count && lane == (i & 31)) {
        const unsigned long long key = make_key(p.noise ? s + p.noise[row * p.E + (long long)id[x] - f.e_base] : s, id[x]);
        if (i < 32) { k0 = key; s0 = s; } else { k1 = key; s1 = s; }
      }
    }
  }
  int r0 = 0, r1 = 0;
  for (int i = 0; i < count; ++i) {
    const unsigned long long o = __shfl_sync(0xffffffffu, i < 32 ? k0 : k1, i & 31);
    r0 += o > k0;
    r1 += o > k1;
  }
  won_key[lane] = 0ull;
  __syncwarp();
  if (k0 && r0 < 32) { won_key[r0] = k0; won_score[r0] = s0; }
  if (k1 && r1 < 32) { won_key[r1] = k1; won_score[r1] = s1; }
  __syncwarp();
  emit_scored(f, row, lane < f.K ? won_key[lane] : 0ull, won_score[lane], lane);
  return true;
}

// A whole block: every landmark the row can see, exactly.  Warp w takes landmarks w, w + 8, ..., four of them in flight.
template <int NP>
__device__ __forceinline__ void scan_row(const SettleParams& p, long long row, unsigned long long (*list)[32], int warp, int lane) {
  const FinalParams& f = p.fin;
  const long long n = row / f.Cq, r = row % f.Cq, seen = min((long long)p.E, p.q_pos0 + r - f.e_base);
  const __nv_bfloat16* kb = f.lk + n * f.kbs;
  const int pieces = f.D >> 3;
  uint4 qv[NP];
  load_row<NP>(qv, f.lq + n * f.qbs + r * f.qrs, pieces, lane);
  unsigned long long m = 0ull, th = 0ull;
  for (long long e0 = warp; e0 < seen; e0 += 4 * SETTLE_WARPS) {
    uint4 kv[4][NP];
    float add[4], acc[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const long long e = min(e0 + x * SETTLE_WARPS, seen - 1);
      load_row<NP>(kv[x], kb + e * f.krs, pieces, lane);
      add[x] = p.noise ? p.noise[row * p.E + e] : 0.f;
    }
    exact_dot4<NP>(acc, qv, kv);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const long long e = e0 + x * SETTLE_WARPS;
      float s = acc[x] * f.scale;
      if (p.noise) s += add[x];
      const unsigned long long key = make_key(s, (unsigned)(f.e_base + e));
      if (e < seen && key > th) {
        list_insert(m, key, lane);
        th = __shfl_sync(0xffffffffu, m, f.K - 1);
      }
    }
  }
  list[warp][lane] = m;
  __syncthreads();
  if (warp == 0) {
    for (int w = 1; w < SETTLE_WARPS; ++w)
      for (int i = 0; i < f.K; ++i) {
        const unsigned long long key = list[w][i];
        if (key <= th) break;                              // lists are descending
        list_insert(m, key, lane);
        th = __shfl_sync(0xffffffffu, m, f.K - 1);
      }
    float clean = from_orderable((unsigned)(m >> 32));
    if (p.noise)
      for (int i = 0; i < f.K; ++i) {
        const unsigned long long key = __shfl_sync(0xffffffffu, m, i);
        const long long e = key ? (long long)(0xffffffffu - (unsigned)key) - f.e_base : 0;
        const float s = exact_dot(f.lq + n * f.qbs + r * f.qrs, kb + e * f.krs, pieces, lane) * f.scale;
        if (lane == i) clean = s;
      }
    emit_scored(f, row, m, clean, lane);
  }
  __syncthreads();
}

// One warp per row; rows whose lists may hide a winner -- more copies of a landmark, or rows of equal scores, than the lists hold -- are
// then scanned by the whole block.  One warp scanning alone, a landmark at a time, was up to 33 times slower than the row scan that
// this path replaces (64 rows x 16,384 landmarks x 768, all rows tied: 13.1 ms against 0.4; now 0.5.  2,080 x 2,080: 1.69 -> 0.67 ms, the row
// scan takes 0.79; 256 x 65,536: 76.7 -> 2.9, 6.1; worst against it: 8 x 260 x 260 x 1,024, 183 us against 121).
template <int NP>
__global__ void __launch_bounds__(SETTLE_WARPS * 32)
lmk_settle_kernel(const __grid_constant__ SettleParams p) {
  __shared__ unsigned long long won_key[SETTLE_WARPS][32];
  __shared__ float won_score[SETTLE_WARPS][32];
  __shared__ int hidden[SETTLE_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long first = (long long)blockIdx.x * p.rows, row = first + warp;
  pdl_trigger();
  pdl_wait();
  bool settled = true;
  if (warp < p.rows && row < p.fin.R) settled = settle_row<NP>(p, row, won_key[warp], won_score[warp], lane);
  if (lane == 0) hidden[warp] = !settled;
  if (__syncthreads_or(!settled))
    for (int w = 0; w < p.rows; ++w)
      if (hidden[w]) scan_row<NP>(p, first + w, won_key, warp, lane);
}

// Landmark ranges per row: enough CTAs to fill the GPU, at most one list per lane of the merging warp.
int screen_lists(const LmkTopkArgs& a, int sms, int* tiles_per_list) {
  const int tiles = (a.E + BN - 1) / BN;
  const long long blocks = (long long)a.N * ((a.Cq + BM - 1) / BM);
  long long lists = (2ll * sms + blocks - 1) / blocks;
  if (lists > MAX_LISTS) lists = MAX_LISTS;
  if (lists > tiles) lists = tiles;
  if (lists < 1) lists = 1;
  *tiles_per_list = (int)((tiles + lists - 1) / lists);
  return (tiles + *tiles_per_list - 1) / *tiles_per_list;
}

}  // namespace

// float32 scores without per-head lists, whole 64-element K steps, room for K + 4 candidates in a warp; below a few thousand pairs
// per sequence the row scan is as fast.
bool lmk_screen_applies(const LmkTopkArgs& a) {
  return a.head_dim == 0 && a.score_round == 0 && a.splits == 0 && a.D % BK == 0 && a.K <= 32 - EXTRA && a.Cq >= 64 && a.E >= 64 &&
         (a.N == 1 || (a.q_batch_stride > 0 && a.k_batch_stride > 0)) && a.q_row_stride > 0 && a.k_row_stride > 0;
}

size_t lmk_screen_workspace_bytes(const LmkTopkArgs& a, int sms) {
  int tpl;
  const size_t lists = (size_t)screen_lists(a, sms, &tpl), rows = (size_t)a.N * a.Cq;
  return align_up(rows * lists * (a.K + EXTRA) * 8, 256) + align_up(rows * lists * 4, 256);
}

int launch_lmk_screen(const LmkTopkArgs& a, void* scratch, int sms, const FinalParams& fin, cudaStream_t stream) {
  ScreenParams p;
  int rc;
  if ((rc = make_rows_map(&p.tm_q, a.lmk_q, a.N, a.Cq, a.D, a.q_row_stride, a.q_batch_stride, BM)) ||
      (rc = make_rows_map(&p.tm_k, a.lmk_k, a.N, a.E, a.D, a.k_row_stride, a.k_batch_stride, BN)))
    return rc;
  p.KC = a.K + EXTRA;
  p.lists = screen_lists(a, sms, &p.tiles_per_list);
  const size_t rows = (size_t)a.N * a.Cq;
  p.part = static_cast<unsigned long long*>(scratch);
  p.eps = reinterpret_cast<float*>(static_cast<char*>(scratch) + align_up(rows * p.lists * p.KC * 8, 256));
  p.noise = a.noise; p.q_pos0 = a.q_pos0; p.e_base = a.e_base;
  p.Cq = a.Cq; p.E = a.E; p.D = a.D; p.scale = fin.scale;
  p.noise_vec = a.E % 4 == 0 && (reinterpret_cast<uintptr_t>(a.noise) & 15u) == 0;
  auto screen = p.KC <= 16 ? lmk_screen_kernel<16> : lmk_screen_kernel<32>;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(screen, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  GCA_CUDA_CHECK(launch_dependent(screen, dim3((unsigned)p.lists, (unsigned)((a.Cq + BM - 1) / BM), (unsigned)a.N), dim3(THREADS), SMEM_BYTES,
                                  stream, p));
  SettleParams sp;
  sp.fin = fin; sp.part = p.part; sp.eps = p.eps; sp.noise = a.noise; sp.q_pos0 = a.q_pos0; sp.KC = p.KC; sp.lists = p.lists; sp.E = a.E;
  // fewer rows than two blocks per SM have warps: blocks of fewer rows, which share a scan among more SMs
  sp.rows = (int)std::min<size_t>(SETTLE_WARPS, (rows + 2 * sms - 1) / (2 * sms));
  const dim3 grid((unsigned)((rows + sp.rows - 1) / sp.rows)), block(SETTLE_WARPS * 32);
  switch ((a.D + 255) / 256) {
    case 1: return (int)launch_dependent(lmk_settle_kernel<1>, grid, block, 0, stream, sp);
    case 2: return (int)launch_dependent(lmk_settle_kernel<2>, grid, block, 0, stream, sp);
    case 3: return (int)launch_dependent(lmk_settle_kernel<3>, grid, block, 0, stream, sp);
    case 4: return (int)launch_dependent(lmk_settle_kernel<4>, grid, block, 0, stream, sp);
    default: return GCA_ERR_SHAPE;
  }
}

}  // namespace gca
