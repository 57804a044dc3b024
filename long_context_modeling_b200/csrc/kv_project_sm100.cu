// Chunk K/V projection fused with the cache append: the two linear maps that turn the chunk
// encoder's output into the chunk cache's K and V (model/DRT.py:770-781 of the reference:
// chunk_k_proj, chunk_v_proj, landmark row cleared) written STRAIGHT into the cache layout at
// the append position (ChunkKVManager.append, model/DRT.py:87-133), and the landmark embeddings
// (the encoder output's last row of every chunk, model/DRT.py:766) copied into the landmark
// cache.  The reference does this as two GEMMs into fresh tensors, two in-place row clears and a
// torch.cat that re-copies the whole cache; here the GEMM's epilogue is the append.
//
//   X  (M = N * count * 64 rows, D columns)  encoder output, bf16, row-major (K-major A operand)
//   Wk, Wv (D x D) bf16 in nn.Linear layout (out, in) = K-major B operand
//   K_cache[n, pos + c, s, :] = X[(n, c, s), :] Wk^T   (zeros for s = 63 when zero_landmark)
//
// tcgen05 GEMM, one CTA per SM, persistent over (row tile, column tile, K|V): two warps issue the TMA copies of a ring of
// 64-deep stages (rows of x, rows of the weights), warp 1 the MMAs into one of two accumulators in tensor memory, eight epilogue warps (two per lane quarter,
// half of the columns each) turn a finished accumulator into bf16 rows of the cache while the next tile is being multiplied;
// the warp that has a chunk's last row also copies it to the landmark cache.  Every wait is bounded
// (GCA_STATUS_TIMEOUT on expiry).
// Tiles (chosen by choose_tile): PAIRS of CTAs on 256 x 256 (cta_group::2) for large products, where each CTA loads half of the
// weight rows: per product a third less shared-memory and L2 traffic than 128 x 256, and power is what a large
// product is bound by (SM clock 1.3-1.6 GHz of 1.97 within milliseconds).  8 x 260 chunks x 64 rows, 768 -> 2 x 768, as the call with the
// allocation of its cache: 252 us after a rest, 289 in a row; cuBLAS, in the same run, 285 / 294 us for the bare product (with
// 128 x 256 tiles in place of pairs the call took 7 % more).  Smaller products take the width of 64, 128, 192 or 256 columns
// whose waves cost least: 6,912 rows 768 -> 768 on 148 SMs are 162 tiles of 256 columns (two waves, the second nearly
// empty) but 216 of 192: 33 -> 19 us.
//
// The same kernel in LINEAR mode is the projection either side of GCA (model/DRT.py:352-355,385):
//   out[m, :] = row_scale[m] * (x[m, :] W^T) + residual[m, :]
// row_scale = 1 / rms(x) turns it into pre-norm RMSNorm + q_proj (the norm's gain is folded into W's
// columns by the caller: RMSNorm(x) W^T = diag(1 / rms) x (W diag(g))^T, so the normalised activations
// are never written), residual makes it o_proj + residual add.  The factors come from the tiles of x as
// they pass (NORM); for pairs, whose tiles arrive on the leader's barriers alone, `row_rms_kernel` reads x
// before.  768 -> 768, 640 / 2,368 / 7,104 rows, x from memory: 6.7 / 8.1 / 14.8 us, with that launch before
// 8.0 / 11.2 / 17.1.  The residual is read two passes of 32 columns ahead of its use; read in the pass itself, an L2 trip each, 1,152 / 3,456 / 7,104 /
// 16,384 rows took 7.3 / 11.4 / 16.1 / 27.4 us, now 6.2 / 9.8 / 14.8 / 25.4.
//
// CROSS-ENTROPY mode is the LM head fused with the loss (model/DRT.py:1055-1064, inference /
// evaluation): the 128 x 256 logit tiles stay in tensor memory, the epilogue reduces each row's tile
// to (maximum, sum of exponentials) and picks out the target's logit, and `ce_combine_kernel`
// merges a row's column tiles into  loss = logsumexp - logit[target].  The (rows x 50,265) logits
// -- 13 GB in bf16 at 8 x 16K tokens -- are never written.
#include "gca_common.cuh"
#include "sm100_ptx.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

#include <type_traits>

namespace gca {

namespace {

using namespace sm100;

constexpr int BM = 128, BK = 64;                      // rows of a CTA's accumulator, K step
constexpr int EPI_WARPS = 8, W_WARP = 2 + EPI_WARPS, NTHREADS = (3 + EPI_WARPS) * 32, STAT_WARPS = 4;

// BN: columns of a tile.  PAIR: two CTAs share a tile of 256 rows (cta_group::2), each loading half of the weight rows.
template <int BN, bool PAIR>
struct Cfg {
  static constexpr int B_ROWS = PAIR ? BN / 2 : BN;
  static constexpr int A_BYTES = BM * BK * 2, STAGE_BYTES = A_BYTES + B_ROWS * BK * 2;
  static constexpr int STAGES = 196608 / STAGE_BYTES;
  static constexpr int OFF_BAR = STAGES * STAGE_BYTES, OFF_SCALE = OFF_BAR + 256, SMEM_BYTES = OFF_SCALE + 2 * BM * 4 + 1024;
  static constexpr int FULL = 0, EMPTY = FULL + STAGES, ACC_FULL = EMPTY + STAGES, ACC_EMPTY = ACC_FULL + 2, SCALE_FULL = ACC_EMPTY + 2,
                       NUM_BARS = SCALE_FULL + 2;
  static constexpr uint32_t IDESC = umma_idesc_bf16(PAIR ? 2 * BM : BM, BN, 0, 0);
  static constexpr int TM = PAIR ? 2 * BM : BM;        // rows of a tile
  static constexpr int ACC_COLS = BN > 128 ? 256 : BN;  // tensor-memory columns of an accumulator
  static_assert(NUM_BARS * 8 + 8 <= 256, "barriers fit their space");
};

struct ProjParams {
  CUtensorMap tm_x, tm_wk, tm_wv;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  int32_t* status;
  long long cache_bs;       // elements between sequences in the caches
  int M, D, rows_per_seq;   // D = contraction length; rows_per_seq = count * 64
  int pos;                  // first chunk position written
  const uint4* x_rows;      // append: x itself and the landmark cache its chunks' last rows go to (or nullptr)
  uint4* lmk;
  long long lmk_bs;         // 16-byte vectors between sequences
  int zero_landmark;
  int wide;                 // output rows start on 32-byte boundaries
  int tiles_m, tiles_n;     // tiles_n = ceil(output columns / BN)
  int nmat;                 // 2: K and V projection with append epilogue; 1: linear mode
  // linear mode: `batches` blocks of M rows, each cut in 64-row blocks (a 128-row tile is two of them, whatever
  // batch they belong to)
  int batches, blocks_per_batch;
  int lead_rows, lead_tiles;          // rows in front of every batch that get the residual alone; copy tiles for them
  long long out_bs, res_bs, scale_bs; // elements (values) between batches
  __nv_bfloat16* out;
  const __nv_bfloat16* residual;      // or nullptr
  const float* row_scale;             // or nullptr
  float rms_eps;                      // NORM: what the rows' mean squares get added
  long long out_stride, res_stride;   // elements between rows
  int ncols;                          // output columns (multiple of 16; any number in cross-entropy mode)
  // cross-entropy mode (linear mode with ce_part != nullptr): the logits never leave tensor memory
  float2* ce_part;                    // (M, tiles_n): running maximum and sum of exp2 of the row's logits in that column tile
  float* ce_target;                   // (M): the target's logit, scaled by log2(e)
  const long long* targets;           // (M) class ids; negative = ignored row
};

// tile t of this CTA -> (which matrix, row tile, column tile)
__device__ __forceinline__ void tile_of(const ProjParams& p, int t, int& which, int& tm, int& tn) {
  tn = t % p.tiles_n;
  const int r = t / p.tiles_n;
  if (p.nmat == 2) { which = r & 1; tm = r >> 1; }
  else { which = 0; tm = r; }
}

// NORM (linear mode, no pairs): the rows are scaled by 1 / rms(x), from the tiles of x as they pass through shared memory: four warps more
// read them beside the MMAs, each thread a row of 64 values, and hand the row's factor to the epilogue.  Every column tile sums its
// rows up again: 16 KB of shared memory per 64-deep stage beside the 24 to 48 KB that the MMAs read.
template <int BN, bool PAIR, bool NORM>
__global__ void __launch_bounds__(NTHREADS + (NORM ? STAT_WARPS * 32 : 0), 1)
kv_project_append_kernel(const __grid_constant__ ProjParams p) {
  static_assert(!(PAIR && NORM), "a pair's tiles arrive on the leader's barriers alone");
  using C = Cfg<BN, PAIR>;
  constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES, A_BYTES = C::A_BYTES, OFF_BAR = C::OFF_BAR, NUM_BARS = C::NUM_BARS;
  constexpr int FULL = C::FULL, EMPTY = C::EMPTY, ACC_FULL = C::ACC_FULL, ACC_EMPTY = C::ACC_EMPTY, SCALE_FULL = C::SCALE_FULL, ACC_COLS = C::ACC_COLS, TMEM_COLS = 2 * ACC_COLS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + NUM_BARS + 1);
  float* scale = reinterpret_cast<float*>(smem + C::OFF_SCALE);           // NORM: [accumulator][row]
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int total = p.tiles_m * p.tiles_n * p.nmat;
  const int ksteps = p.D / BK;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  const int first = PAIR ? blockIdx.x / 2 : blockIdx.x, step = PAIR ? gridDim.x / 2 : gridDim.x;
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&bars[FULL + i], 2); mbar_init(&bars[EMPTY + i], NORM ? 1 + STAT_WARPS : 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars[SCALE_FULL + i], STAT_WARPS); mbar_init(&bars[ACC_FULL + i], 1); mbar_init(&bars[ACC_EMPTY + i], (PAIR ? 2 : 1) * EPI_WARPS); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    if (PAIR) tmem_alloc_pair(tmem_slot, TMEM_COLS);
    else { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&p.tm_x); tma_prefetch_desc(&p.tm_wk); tma_prefetch_desc(&p.tm_wv); }
  tc_fence_before();
  __syncwarp();
  if (PAIR) cluster_sync();
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  pdl_wait();

  if (warp == 0 || warp == W_WARP) {
    // two producers: the rows of x and the rows of the weights, each with its own arrival on FULL (the leader's, for a pair)
    Ring ring; ring.init(STAGES);
    uint32_t issued = 0;
    bool ok = true;
    for (int t = first; t < total && ok; t += step) {
      int which, tm, tn;
      tile_of(p, t, which, tm, tn);
      const CUtensorMap* tw = which ? &p.tm_wv : &p.tm_wk;
      // the CTA's 128 rows in one box, or (several batches) as two 64-row blocks; rows past the end are zero-filled
      int b0 = 0, b1 = 0, r0 = tm * C::TM + (int)rank * BM, r1 = 0;
      const bool blocks = p.batches > 1;
      if (blocks) {
        const int blk = (C::TM / 64) * tm + 2 * (int)rank;
        b0 = blk / p.blocks_per_batch; b1 = (blk + 1) / p.blocks_per_batch;
        r0 = (blk - b0 * p.blocks_per_batch) * 64; r1 = (blk + 1 - b1 * p.blocks_per_batch) * 64;
      }
      for (int ks = 0; ks < ksteps; ++ks) {
        ok = mbar_wait_warp(&bars[EMPTY + ring.st], ring.ph ^ 1, abort_flag, lane);
        if (!ok) break;
        uint8_t* dst = smem + ring.st * STAGE_BYTES;
        uint64_t* full = &bars[FULL + ring.st];
        if (warp == 0) {
          if (rank == 0) mbar_expect_tx_elect(full, (PAIR ? 2 : 1) * A_BYTES);
          if (blocks) {
            tma_load_3d_elect<PAIR>(dst, &p.tm_x, full, ks * BK, r0, b0);
            tma_load_3d_elect<PAIR>(dst + A_BYTES / 2, &p.tm_x, full, ks * BK, r1, b1);
          } else {
            tma_load_2d_elect<PAIR>(dst, &p.tm_x, full, ks * BK, r0);
          }
        } else {
          if (rank == 0) mbar_expect_tx_elect(full, (PAIR ? 2 : 1) * (STAGE_BYTES - A_BYTES));
          tma_load_2d_elect<PAIR>(dst + A_BYTES, tw, full, ks * BK, tn * BN + (int)rank * C::B_ROWS);
        }
        ring.next();
        ++issued;
      }
    }
    if (*abort_flag && rank == 0)          // nothing may land in shared memory after the block (or its pair) has gone
      for (uint32_t back = 0; back < (uint32_t)STAGES && back < issued; ++back) {
        const uint32_t g = issued - 1 - back;
        for (int i = 0; i < (1 << 20); ++i)
          if (mbar_try_wait(&bars[FULL + g % STAGES], (g / STAGES) & 1)) break;
      }
  } else if (warp == 1) {
    // all lanes run the issuing code; elect.sync inside the wrappers picks the issuing lane (of the pair's leader)
    Ring ring; ring.init(STAGES);
    bool ok = true;
    uint32_t tcount = 0;
    for (int t = first; t < total && ok && rank == 0; t += step, ++tcount) {
      const uint32_t ab = tcount & 1;
      ok = mbar_wait_warp(&bars[ACC_EMPTY + ab], ((tcount >> 1) & 1) ^ 1, abort_flag, lane);
      if (ok) tc_fence_after();
      for (int ks = 0; ks < ksteps && ok; ++ks) {
        ok = mbar_wait_warp(&bars[FULL + ring.st], ring.ph, abort_flag, lane);
        if (!ok) break;
        tc_fence_after();
        const uint64_t da = umma_desc_sw128(smem_u32(smem + ring.st * STAGE_BYTES));
        const uint64_t db = umma_desc_sw128(smem_u32(smem + ring.st * STAGE_BYTES + A_BYTES));
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
          if (PAIR) umma_bf16_ss_pair_elect(tmem_base + ab * ACC_COLS, da + kk * 2, db + kk * 2, C::IDESC, (uint32_t)(ks > 0 || kk > 0));
          else umma_bf16_ss_elect(tmem_base + ab * ACC_COLS, da + kk * 2, db + kk * 2, C::IDESC, (uint32_t)(ks > 0 || kk > 0));
        }
        if (PAIR) umma_commit_pair_elect(&bars[EMPTY + ring.st]);
        else umma_commit_elect(&bars[EMPTY + ring.st]);
        ring.next();
      }
      if (ok) {
        if (PAIR) umma_commit_pair_elect(&bars[ACC_FULL + ab]);
        else umma_commit_elect(&bars[ACC_FULL + ab]);
      }
    }
  } else if (NORM && warp > W_WARP) {
    const int row = (warp - W_WARP - 1) * 32 + lane;
    Ring ring; ring.init(STAGES);
    bool ok = true;
    uint32_t tcount = 0;
    for (int t = first; t < total && ok; t += step, ++tcount) {
      float2 sq[4] = {};                                   // eight sums of a row, chains of 8 within a stage and of K / 64 over them: as close to
                                                           // 64 bits as a lane's 24 values and the tree over 32 lanes (4e-8; chains of K / 8 1.1e-7)
      for (int ks = 0; ks < ksteps; ++ks) {
        ok = mbar_wait_warp(&bars[FULL + ring.st], ring.ph, abort_flag, lane);
        if (!ok) break;
        const uint4* x = reinterpret_cast<const uint4*>(smem + ring.st * STAGE_BYTES + row * 128);
        float2 part[4];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 v = x[c ^ (row & 7)];
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
            part[i] = c == 0 ? __fmul2_rn(f, f) : __ffma2_rn(f, f, part[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) sq[i] = __fadd2_rn(sq[i], part[i]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[EMPTY + ring.st]);
        ring.next();
      }
      const uint32_t ab = tcount & 1;
      ok = ok && mbar_wait_warp(&bars[ACC_EMPTY + ab], ((tcount >> 1) & 1) ^ 1, abort_flag, lane);       // the factors before have been read
      if (!ok) break;
      scale[ab * BM + row] = rsqrtf((((sq[0].x + sq[0].y) + (sq[1].x + sq[1].y)) + ((sq[2].x + sq[2].y) + (sq[3].x + sq[3].y))) / (float)p.D + p.rms_eps);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[SCALE_FULL + ab]);
    }
  } else {
    // epilogue: thread = accumulator lane = row of the tile
    const int quad = warp & 3, half = (warp - 2) >> 2;   // warps 2..9: every TMEM lane quarter twice, one half of the columns each
    const int row_in_tile = quad * 32 + lane;
    const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
    auto release = [&](uint32_t ab) {                  // this warp has read its part of the accumulator
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_leader(&bars[ACC_EMPTY + ab]);
        else mbar_arrive(&bars[ACC_EMPTY + ab]);
      }
    };
    bool ok = true;
    uint32_t tcount = 0;
    for (int t = first; t < total + p.lead_tiles && ok; t += step, ++tcount) {
      if (t >= total) {                                  // the lead rows of one batch, 256 columns: residual or zeros
        const int b = (t - total) / p.tiles_n, c0 = (t - total - b * p.tiles_n) * BN, vecs = min(BN, p.ncols - c0) / 8;
        __nv_bfloat16* dst = p.out + b * p.out_bs - p.lead_rows * p.out_stride + c0;
        const __nv_bfloat16* src = p.residual + b * p.res_bs - p.lead_rows * p.res_stride + c0;
        for (int i = ((warp - 2) + EPI_WARPS * (int)rank) * 32 + lane; i < p.lead_rows * vecs; i += (PAIR ? 2 : 1) * EPI_WARPS * 32) {
          const int r = i / vecs, v = i - r * vecs;
          *reinterpret_cast<uint4*>(dst + r * p.out_stride + v * 8) =
              p.residual ? *reinterpret_cast<const uint4*>(src + r * p.res_stride + v * 8) : make_uint4(0, 0, 0, 0);
        }
        continue;
      }
      int which, tm, tn;
      tile_of(p, t, which, tm, tn);
      const uint32_t ab = tcount & 1;
      if (p.nmat == 2 && p.lmk && which == 0 && tn == 0 && half == 0 && (quad & 1)) {
        // the landmark embedding of a chunk is its last row: copied by the warp that has that row
        const long long last = (long long)tm * C::TM + (int)rank * BM + quad * 32 + 31;
        if (last < p.M) {
          const long long n = last / p.rows_per_seq, c = (last - n * p.rows_per_seq) / 64;
          const int vecs = p.D / 8;
          for (int v = lane; v < vecs; v += 32) p.lmk[n * p.lmk_bs + (p.pos + c) * vecs + v] = p.x_rows[last * vecs + v];
        }
      }
      // this thread's row: linear mode out = scale * acc + residual, append mode a cache row (zeros for a landmark row)
      struct Row { __nv_bfloat16* dst; const __nv_bfloat16* res; float sc; bool live, zero; };
      auto row_of = [&] {
        Row o = {nullptr, nullptr, 1.0f, false, false};
        if (p.nmat == 1) {
          const int block = (C::TM / 64) * tm + 2 * (int)rank + (row_in_tile >> 6), b = block / p.blocks_per_batch;
          const long long m = (block - b * p.blocks_per_batch) * 64 + (row_in_tile & 63);
          o.live = b < p.batches && m < p.M;
          if (!NORM && o.live && p.row_scale) o.sc = p.row_scale[b * p.scale_bs + m];
          o.dst = p.out + b * p.out_bs + m * p.out_stride + tn * BN;
          if (o.live && p.residual) o.res = p.residual + b * p.res_bs + m * p.res_stride + tn * BN;
        } else {
          const long long m = (long long)tm * C::TM + (int)rank * BM + row_in_tile;
          o.live = m < p.M;
          const int n = o.live ? (int)(m / p.rows_per_seq) : 0;
          const int r = o.live ? (int)(m - (long long)n * p.rows_per_seq) : 0;       // (chunk, row) inside the appended block
          o.zero = p.zero_landmark && (r & 63) == 63;
          o.dst = (which ? p.v_cache : p.k_cache) + n * p.cache_bs + ((long long)p.pos * 64 + r) * p.D + tn * BN;
        }
        return o;
      };
      // Passes of 32 columns (or the last 16) of one small loop body.  A pass's residual is asked for two passes ahead, that of the first two
      // before the accumulator is waited for.  Not by pairs, whose code the append shares and pays for (8 x 60 chunks, 512 wide, 36.2 -> 36.8 us).
      const int cols = min(BN, p.ncols - tn * BN);       // not every width divides every matrix: the last tile may be a narrow one
      const int c_begin = half * (BN / 2), c_end = min(cols, c_begin + BN / 2);
      const bool ce = p.nmat == 1 && p.ce_part;
      const Row row = ce ? Row{nullptr, nullptr, 1.0f, false, false} : row_of();
      int ask_c = c_begin;
      const bool with_res = p.nmat == 1 && p.residual;
      auto ask = [&](uint4 (&r)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = (row.res && ask_c + 8 * i < c_end) ? *reinterpret_cast<const uint4*>(row.res + ask_c + 8 * i) : make_uint4(0, 0, 0, 0);
        ask_c += 32;
      };
      uint4 rr[4] = {}, rr_next[4];
      if (!PAIR && with_res) { ask(rr); ask(rr_next); }
      ok = mbar_wait_bounded(&bars[ACC_FULL + ab], (tcount >> 1) & 1, abort_flag);
      if (NORM) ok = ok && mbar_wait_bounded(&bars[SCALE_FULL + ab], (tcount >> 1) & 1, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after();
      if (ce) {
        const long long m = (long long)tm * C::TM + (int)rank * BM + row_in_tile;
        const bool live = m < p.M;
        if (half) { release(ab); continue; }             // a row's tile is reduced by one thread
        // cross-entropy mode: per row, the maximum and the sum of exponentials of this column
        // tile's logits (base 2, logits scaled by log2 e) and the target's logit if it lies here
        const float sc = ((live && p.row_scale) ? p.row_scale[m] : 1.0f) * GCA_LOG2E;
        const long long tgt = live ? p.targets[m] - (long long)tn * BN : -1;
        float mx = -INFINITY, sum = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < cols; c0 += 16) {
          uint32_t v[16];
          tmem_ld_32x32b_x16(tlane + ab * ACC_COLS + c0, v);
          tmem_ld_wait();
          float x[16];
          float pm = -INFINITY;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            x[i] = (c0 + i < cols) ? __uint_as_float(v[i]) * sc : -INFINITY;
            pm = fmaxf(pm, x[i]);
          }
          if (tgt >= c0 && tgt < c0 + 16 && tgt < cols) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (tgt == c0 + i) p.ce_target[m] = x[i];
          }
          const float nm = fmaxf(mx, pm);
          float ps = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) ps += ex2_approx(x[i] - nm);
          sum = sum * ex2_approx(mx - nm) + ps;
          mx = nm;
        }
        if (live) p.ce_part[m * p.tiles_n + tn] = make_float2(mx, sum);
        release(ab);
        continue;
      }
      const float sc = NORM ? scale[ab * BM + row_in_tile] : row.sc;
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 32) {
        uint32_t v[32], w[16];
        const bool two = c0 + 16 < c_end;
        if (PAIR && with_res) { ask_c = c0; ask(rr); }
        tmem_ld_32x32b_x32(tlane + ab * ACC_COLS + c0, v);
        const uint32_t rw[16] = {rr[0].x, rr[0].y, rr[0].z, rr[0].w, rr[1].x, rr[1].y, rr[1].z, rr[1].w,
                                 rr[2].x, rr[2].y, rr[2].z, rr[2].w, rr[3].x, rr[3].y, rr[3].z, rr[3].w};
        tmem_ld_wait();
        if (row.zero) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
          w[i] = pack_bf16x2(fmaf(__uint_as_float(v[2 * i]), sc, __uint_as_float(rw[i] << 16)),
                             fmaf(__uint_as_float(v[2 * i + 1]), sc, __uint_as_float(rw[i] & 0xffff0000u)));
        if (!PAIR && with_res) {
#pragma unroll
          for (int i = 0; i < 4; ++i) rr[i] = rr_next[i];
          ask(rr_next);
        }
        if (!row.live) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h && !two) break;
          __nv_bfloat16* dst = row.dst + c0 + 16 * h;
          if (p.wide) st_global_256(dst, w[8 * h], w[8 * h + 1], w[8 * h + 2], w[8 * h + 3], w[8 * h + 4], w[8 * h + 5], w[8 * h + 6], w[8 * h + 7]);
          else {
            reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[8 * h], w[8 * h + 1], w[8 * h + 2], w[8 * h + 3]);
            reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[8 * h + 4], w[8 * h + 5], w[8 * h + 6], w[8 * h + 7]);
          }
        }
      }
      release(ab);
    }
  }
  tc_fence_before();
  __syncwarp();
  if (PAIR) cluster_sync();                            // neither CTA leaves while the other's MMAs or arrivals may touch it
  else __syncthreads();
  if (warp == 1) {
    if (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicOr(p.status, GCA_STATUS_TIMEOUT);
}

// row_scale[m] = rsqrt(mean(x[m, :]^2) + eps): one warp per row, 16-byte loads; blockIdx.y: batch.
__global__ void row_rms_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ row_scale, long long M, int D,
                               long long stride, float eps, long long x_bs, long long scale_bs) {
  const long long m = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= M) return;
  const int lane = threadIdx.x & 31;
  const uint4* row = reinterpret_cast<const uint4*>(x + blockIdx.y * x_bs + m * stride);
  row_scale += blockIdx.y * scale_bs;
  float acc = 0.f;
  for (int i = lane; i < D / 8; i += 32) {
    const uint4 v = row[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      acc = fmaf(a, a, acc); acc = fmaf(b, b, acc);
    }
  }
#pragma unroll
  for (int of = 16; of > 0; of >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, of);
  if (lane == 0) row_scale[m] = rsqrtf(acc / (float)D + eps);
}

// out[m, c] = silu(gu[m, c]) * gu[m, I + c]: the activation between one gate|up product and down_proj
// (the reference's fused SwiGLU, model/llama.py:290-300).  One thread per 8 columns, 16-byte accesses.
__global__ void silu_mul_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, long long M, int I,
                                long long in_stride, long long out_stride) {
  const int per_row = I / 8;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= M * per_row) return;
  const long long m = t / per_row;
  const int c = (int)(t - m * per_row) * 8;
  const uint4 g = *reinterpret_cast<const uint4*>(gu + m * in_stride + c);
  const uint4 u = *reinterpret_cast<const uint4*>(gu + m * in_stride + I + c);
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float g0 = __uint_as_float(gw[j] << 16), g1 = __uint_as_float(gw[j] & 0xffff0000u);
    const float u0 = __uint_as_float(uw[j] << 16), u1 = __uint_as_float(uw[j] & 0xffff0000u);
    const __nv_bfloat162 b = __floats2bfloat162_rn(g0 / (1.f + __expf(-g0)) * u0, g1 / (1.f + __expf(-g1)) * u1);
    o[j] = *reinterpret_cast<const uint32_t*>(&b);
  }
  *reinterpret_cast<uint4*>(out + m * out_stride + c) = make_uint4(o[0], o[1], o[2], o[3]);
}

// loss[m] = ln(sum_j exp(logit_j)) - logit_target from the per-tile partials (base 2 inside); ignored rows: 0.
__global__ void ce_combine_kernel(const float2* __restrict__ part, const float* __restrict__ tlogit, const long long* __restrict__ targets,
                                  float* __restrict__ loss, float* __restrict__ lse_out, long long M, int tiles) {
  const long long m = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= M) return;
  const int lane = threadIdx.x & 31;
  float mx = -INFINITY, sum = 0.f;
  for (int t = lane; t < tiles; t += 32) {
    const float2 v = part[m * tiles + t];
    const float nm = fmaxf(mx, v.x);
    sum = sum * (mx == -INFINITY ? 0.f : exp2f(mx - nm)) + v.y * (v.x == -INFINITY ? 0.f : exp2f(v.x - nm));
    mx = nm;
  }
#pragma unroll
  for (int of = 16; of > 0; of >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, mx, of), os = __shfl_xor_sync(0xffffffffu, sum, of);
    const float nm = fmaxf(mx, om);
    sum = sum * (mx == -INFINITY ? 0.f : exp2f(mx - nm)) + os * (om == -INFINITY ? 0.f : exp2f(om - nm));
    mx = nm;
  }
  if (lane == 0) {
    const float lse2 = mx + log2f(sum);                        // base-2 log-sum-exp of the scaled logits
    const float ln2 = 0.6931471805599453f;
    if (lse_out) lse_out[m] = lse2 * ln2;
    loss[m] = targets[m] >= 0 ? (lse2 - tlogit[m]) * ln2 : 0.f;
  }
}

}  // namespace

int launch_skinny_linear(const LinearArgs& a, float rms_eps, cudaStream_t stream);
bool few_rows(long long M, int N, int K, bool with_norm, int sms);

namespace {

// Which tile: the width, or the pairs, whose waves cost least.
//   APPEND (and cross-entropy): in units of column-steps of one CTA a tile costs its width plus ~64 for its prologue and epilogue tail; wide pairs, which read
// the least shared memory and L2 per product, ~48 (power is what a large product runs into).
//   The linear products, in ns: once, a wave, and a wave's stage (64 of K), fitted to 1,400 to 1,600 sizes of each (300 to 131,072 rows, 256 to 4,096 columns,
// K 128 to 4,096, x from memory).  The choice is the fastest of the five or within 0.3 % of it on average, 5 % in 99 of 100.  A residual costs pairs more, which read
// it in the pass itself: 24,576 rows 2,048 -> 1,024 take pairs with one (74.7 us, 256 columns 91.4, 128 columns 98.8) and without, 12,288 rows 768 -> 2,048
// only without (34.3, 256 columns 38.2; with a residual 51.5, 192 columns 47.2).  NORM: every column tile sums up the factors from the tiles of x again; for pairs a
// launch before reads x (0.75 ns for 64 x 64 values of it): 24,576 rows 768 -> 4,096 121.1 us, 256 columns 144.4, but 3,072 -> 256 66.0 and 52.3.
enum class Product { APPEND, PLAIN, RESIDUAL, NORM };
struct TileChoice { int bn; bool pair; };
struct TileCost { TileChoice tile; int once, wave, stage; };
constexpr TileCost TILE_COSTS[4][5] = {
    {{{256, true}, 0, 304, 0}, {{256, false}, 0, 320, 0}, {{192, false}, 0, 256, 0}, {{128, false}, 0, 192, 0}, {{64, false}, 0, 128, 0}},
    {{{256, true}, 1100, 2440, 275}, {{256, false}, 600, 1610, 371}, {{192, false}, 500, 1110, 332}, {{128, false}, 110, 1050, 223}, {{64, false}, 0, 560, 197}},
    {{{256, true}, 2510, 5180, 216}, {{256, false}, 690, 3910, 329}, {{192, false}, 450, 2390, 289}, {{128, false}, 0, 1700, 238}, {{64, false}, 40, 1010, 153}},
    {{{256, true}, 2900, 2470, 318}, {{256, false}, 600, 2240, 398}, {{192, false}, 130, 1870, 377}, {{128, false}, 560, 1230, 361}, {{64, false}, 90, 750, 320}}};
TileChoice choose_tile(Product product, long long rows64, int ncols, int k, int nmat, int sms) {
  auto ceil_div = [](long long a, long long b) { return (a + b - 1) / b; };
  TileChoice best = {};
  long long best_cost = -1;
  for (const TileCost& c : TILE_COSTS[(int)product]) {
    const long long tiles = ceil_div(rows64, c.tile.pair ? 4 : 2) * ceil_div(ncols, c.tile.bn) * nmat;
    const long long factors = product == Product::NORM && c.tile.pair ? rows64 * (k / BK) * 3 / 4 : 0;
    const long long cost = c.once + factors + ceil_div(tiles, c.tile.pair ? sms / 2 : sms) * (c.wave + (long long)(k / BK) * c.stage);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = c.tile; }
  }
  return best;
}

template <int BN, bool PAIR, bool NORM>
int launch_tiles(const ProjParams& p, int sms, cudaStream_t stream) {
  using C = Cfg<BN, PAIR>;
  auto kernel = kv_project_append_kernel<BN, PAIR, NORM>;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
  const long long tiles = (long long)p.tiles_m * p.tiles_n * p.nmat + p.lead_tiles;
  const dim3 block(NTHREADS + (NORM ? STAT_WARPS * 32 : 0));
  if (PAIR) {
    const unsigned pairs = (unsigned)(tiles < sms / 2 ? tiles : sms / 2);
    return (int)launch_dependent_pairs(kernel, dim3(2 * pairs), block, C::SMEM_BYTES, stream, p);
  }
  return (int)launch_dependent(kernel, dim3((unsigned)(tiles < sms ? tiles : sms)), block, C::SMEM_BYTES, stream, p);
}

// rows64: 64-row blocks of x (of all batches).  Fills in the tile counts; the weight maps are made here because their box is the tile's.
int launch_product(ProjParams& p, const void* wk, const void* wv, long long w_stride, long long rows64, TileChoice tile, int sms, cudaStream_t stream,
                   bool norm = false) {
  const int tm = tile.pair ? 4 : 2, box = tile.pair ? tile.bn / 2 : tile.bn;
  int rc;
  if ((rc = make_matrix_map(&p.tm_wk, wk, p.ncols, p.D, w_stride, box)) || (rc = make_matrix_map(&p.tm_wv, wv, p.ncols, p.D, w_stride, box))) return rc;
  p.tiles_m = (int)((rows64 + tm - 1) / tm);
  p.tiles_n = (p.ncols + tile.bn - 1) / tile.bn;
  p.lead_tiles = p.lead_rows > 0 ? p.batches * p.tiles_n : 0;
  if ((long long)p.tiles_m * p.tiles_n * p.nmat + p.lead_tiles >= (1ll << 30)) return GCA_ERR_TOO_LARGE;
  auto width = [&](auto with) {
    constexpr bool NORM = decltype(with)::value;
    if (tile.bn == 256) return launch_tiles<256, false, NORM>(p, sms, stream);
    if (tile.bn == 192) return launch_tiles<192, false, NORM>(p, sms, stream);
    if (tile.bn == 128) return launch_tiles<128, false, NORM>(p, sms, stream);
    return launch_tiles<64, false, NORM>(p, sms, stream);
  };
  if (tile.pair) return launch_tiles<256, true, false>(p, sms, stream);
  return norm ? width(std::true_type()) : width(std::false_type());
}

}  // namespace

int launch_linear_ce(const LinearCeArgs& a, int sms, cudaStream_t stream) {
  ProjParams p;
  if (a.M >= (1ll << 31)) return GCA_ERR_TOO_LARGE;
  int rc;
  if ((rc = make_matrix_map(&p.tm_x, a.x, a.M, a.K, a.x_stride, BM))) return rc;
  p.k_cache = p.v_cache = nullptr; p.status = a.status; p.cache_bs = 0;
  p.M = (int)a.M; p.D = a.K; p.rows_per_seq = 1; p.pos = 0; p.zero_landmark = 0; p.nmat = 1;
  p.out = nullptr; p.residual = nullptr; p.row_scale = a.row_scale; p.out_stride = p.res_stride = 0; p.ncols = a.N;
  p.batches = 1; p.blocks_per_batch = 0; p.lead_rows = 0; p.out_bs = p.res_bs = p.scale_bs = 0;
  // workspace: partials (M, 256-column tiles) float2, then the target logits (M) float
  const long long tiles = (a.N + 255) / 256;
  p.ce_part = reinterpret_cast<float2*>(a.workspace);
  p.ce_target = reinterpret_cast<float*>(p.ce_part + a.M * tiles);
  p.targets = reinterpret_cast<const long long*>(a.targets);
  TileChoice tile = choose_tile(Product::APPEND, (a.M + 63) / 64, a.N, a.K, 1, sms);
  tile.bn = 256;                                       // the workspace counts 256-column tiles
  if ((rc = launch_product(p, a.w, a.w, a.w_stride, (a.M + 63) / 64, tile, sms, stream))) return rc;
  const int warps = 8;
  ce_combine_kernel<<<(unsigned)((a.M + warps - 1) / warps), warps * 32, 0, stream>>>(p.ce_part, p.ce_target, p.targets, a.loss, a.lse, a.M,
                                                                                    p.tiles_n);
  return (int)cudaGetLastError();
}

int launch_row_rms(const RowRmsArgs& a, cudaStream_t stream) {
  if (a.M == 0) return 0;
  const int warps = 8;
  row_rms_kernel<<<(unsigned)((a.M + warps - 1) / warps), warps * 32, 0, stream>>>(
      (const __nv_bfloat16*)a.x, a.row_scale, a.M, a.D, a.x_stride, a.eps, 0, 0);
  return (int)cudaGetLastError();
}

int launch_silu_mul(const void* gu, void* out, long long M, int I, long long in_stride, long long out_stride, cudaStream_t stream) {
  const long long threads = M * (I / 8);
  if (threads == 0) return 0;
  silu_mul_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>((const __nv_bfloat16*)gu, (__nv_bfloat16*)out, M, I, in_stride,
                                                                            out_stride);
  return (int)cudaGetLastError();
}

// norm_scratch: nullptr, or where the rows' factors 1 / rms(x) may be put, batches x M values, one.row_scale being NULL.
int launch_linear(const LinearBatchedArgs& ba, float* norm_scratch, int sms, cudaStream_t stream) {
  LinearBatchedArgs args = ba;
  LinearArgs& a = args.one;
  const float norm_eps = args.rms_eps;
  if (norm_scratch) { args.rms_eps = 0.f; args.scale_batch_stride = a.M; }
  // batches that lie back to back are one block of rows
  if (args.batches > 1 && args.lead_rows == 0 && args.x_batch_stride == a.M * a.x_stride && args.out_batch_stride == a.M * a.out_stride &&
      (!a.residual || args.residual_batch_stride == a.M * a.residual_stride) && (!a.row_scale || args.scale_batch_stride == a.M)) {
    a.M *= args.batches;
    args.batches = 1;
  }
  auto factors = [&]() -> int {                          // by a launch of their own
    if (args.batches > 65535) return GCA_ERR_TOO_LARGE;
    const int warps = 8;
    row_rms_kernel<<<dim3((unsigned)((a.M + warps - 1) / warps), (unsigned)args.batches), warps * 32, 0, stream>>>(
        (const __nv_bfloat16*)a.x, norm_scratch, a.M, a.K, a.x_stride, norm_eps, args.x_batch_stride, args.scale_batch_stride);
    return (int)cudaGetLastError();
  };
  if (args.batches == 1 && args.lead_rows == 0 && a.M <= GCA_SKINNY_ROWS && (args.rms_eps > 0.f || few_rows(a.M, a.N, a.K, false, sms))) {
    if (norm_scratch) {
      if (int rc = factors()) return rc;
      a.row_scale = norm_scratch;
    }
    return launch_skinny_linear(a, args.rms_eps, stream);
  }
  if (args.rms_eps > 0.f) return GCA_ERR_SHAPE;
  ProjParams p;
  if (a.M >= (1ll << 31)) return GCA_ERR_TOO_LARGE;
  int rc;
  rc = args.batches > 1 ? make_rows_map(&p.tm_x, a.x, args.batches, a.M, a.K, a.x_stride, args.x_batch_stride, 64)
                        : make_matrix_map(&p.tm_x, a.x, a.M, a.K, a.x_stride, BM);
  if (rc) return rc;
  p.k_cache = p.v_cache = nullptr; p.status = a.status; p.cache_bs = 0;
  const long long per_batch = (a.M + 63) / 64;
  p.M = (int)a.M; p.D = a.K; p.rows_per_seq = 1; p.pos = 0; p.zero_landmark = 0; p.nmat = 1;
  p.batches = args.batches; p.blocks_per_batch = (int)per_batch; p.lead_rows = args.lead_rows;
  p.out_bs = args.out_batch_stride; p.res_bs = args.residual_batch_stride; p.scale_bs = args.scale_batch_stride;
  p.out = (__nv_bfloat16*)a.out; p.residual = (const __nv_bfloat16*)a.residual; p.row_scale = a.row_scale;
  p.out_stride = a.out_stride; p.res_stride = a.residual_stride; p.ncols = a.N;
  p.wide = (reinterpret_cast<uintptr_t>(a.out) & 31u) == 0 && a.out_stride % 16 == 0 && args.out_batch_stride % 16 == 0;
  p.ce_part = nullptr; p.ce_target = nullptr; p.targets = nullptr;
  const long long blocks = per_batch * args.batches;
  if (blocks >= (1ll << 30)) return GCA_ERR_TOO_LARGE;
  const TileChoice tile = choose_tile(norm_scratch ? Product::NORM : a.residual ? Product::RESIDUAL : Product::PLAIN, blocks, a.N, a.K, 1, sms);
  const bool norm = norm_scratch && !tile.pair;
  p.rms_eps = norm_eps;
  if (norm_scratch && !norm) {
    if ((rc = factors())) return rc;
    p.row_scale = norm_scratch;
  }
  return launch_product(p, a.w, a.w, a.w_stride, blocks, tile, sms, stream, norm);
}

int launch_kv_project_append(const KvProjectArgs& a, int sms, cudaStream_t stream) {
  ProjParams p;
  const long long M = (long long)a.N * a.count * 64;
  int rc;
  if ((rc = make_matrix_map(&p.tm_x, a.x, M, a.D, a.D, BM))) return rc;
  p.k_cache = (__nv_bfloat16*)a.k_cache; p.v_cache = (__nv_bfloat16*)a.v_cache; p.status = a.status;
  p.cache_bs = a.cache_batch_stride; p.M = (int)M; p.D = a.D; p.rows_per_seq = a.count * 64; p.pos = a.pos;
  p.zero_landmark = a.zero_landmark; p.nmat = 2;
  p.out = nullptr; p.residual = nullptr; p.row_scale = nullptr; p.out_stride = p.res_stride = 0; p.ncols = a.D;
  p.ce_part = nullptr; p.ce_target = nullptr; p.targets = nullptr;
  p.batches = 1; p.blocks_per_batch = 0; p.lead_rows = 0; p.out_bs = p.res_bs = p.scale_bs = 0;
  p.wide = 1;                                          // the entry point asks for 32-byte aligned caches
  p.x_rows = (const uint4*)a.x; p.lmk = (uint4*)a.lmk_cache; p.lmk_bs = a.lmk_cache_batch_stride / 8;
  return launch_product(p, a.wk, a.wv, a.D, M / 64, choose_tile(Product::APPEND, M / 64, a.D, a.D, 2, sms), sms, stream);
}

}  // namespace gca
