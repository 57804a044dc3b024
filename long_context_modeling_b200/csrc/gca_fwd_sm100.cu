// GCA forward on the 5th-generation tensor cores (tcgen05 + TMEM), bf16, S = L = D = 64.
//
// Work unit: one (sequence n, query chunk j, PAIR of q heads A, B).  Every product is per head with 64-row MMAs:
//
//   S  = Q K^T     M = 64, N = 64, K = 64, head A in lanes 0-15 of every 32-lane quarter of tensor memory, head B in lanes 16-31 of
//                  the same columns
//   O += P V       P is the A operand straight from tensor memory, V an MN-major B operand
//
// so S of a pair takes 64 columns and O another 64: three S accumulators, two O accumulators and three P operands fit.  (Stacked
// 128-row products of both heads take the same tensor time, half of their result being thrown away, but 128 columns each: with
// one O accumulator the unit's output had to be written before the next unit's products could start.)
//
// Per retrieved slot k (padding slots are skipped):  S -> one thread per row computes
// P = (w_k / l) * exp2(S c - m) in bf16 (no running rescale: a slot's softmax spans exactly
// one key tile) -> O accumulates over all K slots in ONE TMEM tile (fused weighted merge).
// K_k / V_k tiles for both heads arrive with ONE TMA copy each, straight from the chunk
// cache with the retrieved chunk index as a tensor coordinate (no gathered copy exists).
//
// CTA = 16 warps.
//   warps 0-11  three softmax warpgroups (thread = TMEM lane = row); slot g of the CTA belongs to group g % 3, which has an S
//               accumulator and a P operand of its own, so one group's chain S -> TMEM read -> exp2 -> P -> PV overlaps the others'
//   warp  12    walks the unit list, publishes one RECORD per valid slot in shared memory, issues the TMA copies of Q and K
//   warp  13    TMA producer for V (separate ring; K is released as soon as S is done)
//   warp  14    issues the S MMAs;  warp 15 the PV MMAs (one O accumulator per unit, slots in order, so
//               the result does not depend on timing)
// All other roles follow the records, slot by slot, and have no code that runs once per unit: that code is never in the instruction
// cache and costs a warp ~10 cycles an instruction (an event trace of the form with one descriptor per unit: 1,500 cycles between
// a group's last slot of a unit and its first of the next, of ~10,000 per unit).
// 12 heads: 8 x 256 chunks, K = 8: 390 -> 357 us (345 to 352 with the polling loops out of line), 1 x 1,024, K = 16: 389 -> 364 (353 to 368).  Tried on this form and slower: Q in tensor
// memory so that both issuers run one code (363), one copy of the output code (357), the next record and the
// next barriers probed in the middle of a slot (398 us: what counts is how many barrier operations there are, not where their
// latency falls), probes by one elected lane (+9 %), a fourth softmax group (+28 %, with registers moved to it from the other warps).
// Ring stages are released by tcgen05.commit straight onto the producers' barriers.  CTAs are persistent and
// walk the units in an order (late_chunks_first) in which concurrently running CTAs touch the cache
// of few sequences (L2 reuse of chunks retrieved many times).  Every mbarrier wait is bounded;
// on expiry the CTA flags GCA_STATUS_TIMEOUT, drains its copies and unwinds.
#include <cstdlib>

#define GCA_WAIT_OUT_OF_LINE          // 358 -> 345 us, 1 x 1,024 chunks, K = 16: 364 -> 353; slower in the other kernels
#include "gca_common.cuh"
#include "sm100_ptx.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

namespace gca {

namespace {

using namespace sm100;

constexpr int TILE_BYTES = 64 * 64 * 2;
constexpr int PAIR_BYTES = 2 * TILE_BYTES;
constexpr int NWG = 3;                      // softmax warpgroups
constexpr int NK = 6, NV = 6;               // K / V ring stages
constexpr int NR = 18;                      // slot records
constexpr int NTHREADS = (4 * NWG + 4) * 32;
constexpr int KPROD_WARP = 4 * NWG, VPROD_WARP = KPROD_WARP + 1, SMMA_WARP = KPROD_WARP + 2;   // last warp: PV issuer
// Tensor memory: S0 S1 S2 (64 columns each; group w has S w) | O0 O1 (64 each; unit u uses O u % 2) | P0 P1 P2 (32 each).  P -- the bf16
// probabilities, one row per lane, two values per column -- never goes through shared memory, whose 128 bytes per clock
// (operand reads of the MMAs + TMA writes) are the kernel's tightest resource.
constexpr int TMEM_COLS = 512;
constexpr int TMEM_O = NWG * 64, TMEM_P = TMEM_O + 2 * 64;
constexpr uint32_t LANE16 = 16u << 16;      // lane offset of head B's 64-row tile

// What the other roles need to know about a slot.  The warp that issues the Q / K copies walks the unit list, reads the retrieved
// indices and weights, does all the index and address arithmetic once and publishes the result here.
struct SlotRec {
  uint32_t flags;           // REC_*
  float w;                  // retrieval weight
  long long lse_off;        // element offset of (unit, head A, this slot, row 0) in lse
  long long out_off;        // element offset of (unit, head A, row 0) in out
  uint32_t unit;            // running number of the unit in this CTA
  int32_t hk0, n, chunk;    // tensor coordinates of the V copy: kv head, sequence, chunk
  int32_t pad[2];
};
constexpr uint32_t REC_END = 1, REC_FIRST = 2, REC_LAST = 4, REC_TWO = 8, REC_SHARE = 16;     // END: no more slots; FIRST / LAST of its unit
static_assert(sizeof(SlotRec) == 48, "slot record");

constexpr int OFF_Q = 0;                              // [2 bufs][A B]
constexpr int OFF_K = OFF_Q + 2 * PAIR_BYTES;         // [NK][A B]
constexpr int OFF_V = OFF_K + NK * PAIR_BYTES;        // [NV][A B]
constexpr int OFF_BAR = OFF_V + NV * PAIR_BYTES;
constexpr int OFF_REC = OFF_BAR + 512;                // [NR]
constexpr int SMEM_BYTES = OFF_REC + NR * 48 + 1024;  // + alignment slack

// Barriers.
//   REC_FULL[r]    record of slot g, r = g % 18, is written (1 arrival).  Its place is written again for slot g + 18, which needs S of slot
//                  g + 12 complete, hence S of g + 9 read, hence P of g + 6 written, hence PV of g + 3 complete: every role is past g
//   K_FULL[stage]  the slot's K tile has landed (producer's expect_tx arrival + bytes) AND the S
//                  accumulator the slot will use has been read by the group that had it three slots
//                  earlier (its 4 warps arrive here)
//   S_FULL[group]  S of the group's next slot is complete (commit)
//   K_EMPTY[stage] same commit, for the K producer
//   V_FULL[stage]  the V tile has landed AND the slot's group has written P; the PV issuer's only wait
//   P_EMPTY[group] PV of the group's latest slot is complete (commit): its P region may be rewritten
//   V_EMPTY[stage] same commit, for the V producer
//   O_FULL[b]      the unit that uses accumulator b is complete (waited for only by who has seen P_EMPTY of the unit's last slot, so it
//                  is never more than this phase behind); O_EMPTY[b]: it has been read
// A barrier that belongs to a group completes one phase per slot of that group, and the next
// phase cannot complete before the group has acted on this one.
enum Bar { Q_FULL = 0, Q_EMPTY = 2, K_FULL = 4, K_EMPTY = K_FULL + NK, V_FULL = K_EMPTY + NK, V_EMPTY = V_FULL + NV,
           S_FULL = V_EMPTY + NV, P_EMPTY = S_FULL + NWG, O_FULL = P_EMPTY + NWG, O_EMPTY = O_FULL + 2, REC_FULL = O_EMPTY + 2,
           NUM_BARS = REC_FULL + NR };
static_assert(NUM_BARS * 8 + 16 <= 512, "barrier block");
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

struct FwdTcParams {
  CUtensorMap tm_q, tm_k2, tm_v2, tm_k1, tm_v1;   // *2: both heads of a pair per copy, *1: one head
  const int32_t* indices;
  const float* weights;
  __nv_bfloat16* out;
  float* lse;
  int32_t* status;
  long long* prof;          // optional cycle counters of block 0 (debug), or nullptr
  long long os[4];
  int units;
  int N, J, Hq, Hkv, G, K, C, HP;
  bool late_first;           // order of the units, see row_block_at
  int pair;                 // 1: a unit is a pair of q heads; 0: a single head (GCA_ALGO_TC_UNPAIRED)
  int dbg;                  // profile builds only: bit mask of work to skip (timing experiments)
  int wide_store;           // every output row is 32-byte aligned: 256-bit stores
  float c2;
  float off_by_one;
};

// Debug tracing (compiled in only with -DGCA_PROFILE).
#ifdef GCA_PROFILE
// event trace of block 0: prof[64 + event * 256 + slot] = clock of that event for that slot
#define GCA_TRACE(ev, slot) do { if (p.prof != nullptr && blockIdx.x == 0 && (slot) < 256u) p.prof[64 + (ev) * 256 + (slot)] = clock64(); } while (0)
#else
#define GCA_TRACE(ev, slot) do { } while (0)
#endif

// Timing experiments (compiled in only with -DGCA_DBGKNOBS): skip parts of the work.
#ifdef GCA_DBGKNOBS
#define GCA_DBG(bit) ((p.dbg >> (bit)) & 1)
#else
#define GCA_DBG(bit) 0
#endif

struct UnitInfo { int h0, hk0; bool two, share; };
__device__ __forceinline__ UnitInfo unit_info(const FwdTcParams& p, int hp) {
  UnitInfo t;
  t.h0 = p.pair ? 2 * hp : hp;
  t.two = p.pair && (t.h0 + 1) < p.Hq;
  if (p.G == 1) { t.hk0 = t.h0; t.share = false; }
  else { t.hk0 = t.h0 / p.G; t.share = t.two && ((t.h0 + 1) / p.G == t.hk0); }
  return t;
}
// Lane-parallel read of one row of retrieved indices (the Q / K producer, one row ahead).
__device__ __forceinline__ int load_index_row(const FwdTcParams& p, int u, int zj, int lane) {
  if (u >= p.units || lane >= p.K) return -1;
  return slot_chunk(p.indices, zj, p.K, lane);
}
__device__ __forceinline__ unsigned valid_mask(const FwdTcParams& p, int idx) {
  return __ballot_sync(0xffffffffu, idx >= 0 && idx < p.C);
}

__device__ __forceinline__ SlotRec* slot_recs(uint8_t* smem) { return reinterpret_cast<SlotRec*>(smem + OFF_REC); }

// Bounded wait (one lane) for the copies of a ring that may still be in flight: no bulk copy
// may land in shared memory after the CTA has exited.
__device__ __forceinline__ void drain_ring(uint64_t* bars, int full0, uint32_t issued, int depth) {
  for (uint32_t back = 0; back < (uint32_t)depth && back < issued; ++back) {
    const uint32_t g = issued - 1 - back;
    for (int i = 0; i < (1 << 20); ++i)
      if (mbar_try_wait(&bars[full0 + g % depth], (g / depth) & 1)) break;
  }
}

// ----------------------------------------------------------------------------- Q / K producer
// Walks this CTA's units; lane k publishes the record of slot k and issues its K copy when its turn has come, the first valid lane the
// unit's Q copy too.  Everything a unit needs that no slot will write is
// also done here (rare: the first K chunks of a sequence): zero output rows of a unit without
// valid slots, zero lse of padding slots, the bad-index status bit.
__device__ void kproducer_role(const FwdTcParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int lane) {
  SlotRec* recs = slot_recs(smem);
  PairCursor c;
  c.init(p.HP);
  Ring ring; ring.init(NK);
  Ring rr; rr.init(NR);
  uint32_t un = 0, issued = 0, q_issued = 0;
  bool ok = true;
  const unsigned full = (p.K >= 32) ? 0xffffffffu : ((1u << p.K) - 1u);
  int next_zj = row_block_at(c.outer, p.N, p.J, p.late_first);
  int next_idx = load_index_row(p, c.u, next_zj, lane);
  float next_w = (c.u < p.units && lane < p.K) ? p.weights[(long long)next_zj * p.K + lane] : 0.f;
  for (; c.u < p.units && ok; c.advance()) {
    const int zj = next_zj, my_idx = next_idx;
    const float my_w = next_w;
    next_zj = row_block_at(c.next_outer(), p.N, p.J, p.late_first);
    next_idx = load_index_row(p, c.u + gridDim.x, next_zj, lane);
    next_w = (c.u + gridDim.x < p.units && lane < p.K) ? p.weights[(long long)next_zj * p.K + lane] : 0.f;
    const unsigned mask = valid_mask(p, my_idx);
    const UnitInfo t = unit_info(p, c.inner);
    const int n = zj / p.J, j = zj - n * p.J;
    const long long lse_off = ((long long)zj * p.Hq + t.h0) * p.K * 64;
    const long long out_off = n * p.os[0] + j * p.os[1] + t.h0 * p.os[2];
    if (__any_sync(0xffffffffu, my_idx >= p.C) && p.status && lane == 0) atomicOr(p.status, GCA_STATUS_BAD_INDEX);
    if (mask != full) {
      const int rows = t.two ? 128 : 64;                       // rows of the unit: head A, then head B
      if (p.lse)
        for (int k = 0; k < p.K; ++k)
          if (!((mask >> k) & 1))
            for (int i = lane; i < rows; i += 32) p.lse[lse_off + ((long long)(i >> 6) * p.K + k) * 64 + (i & 63)] = 0.f;
      if (mask == 0) {
        for (int i = lane; i < rows * 8; i += 32) {
          const int r = i >> 3;
          reinterpret_cast<uint4*>(p.out + out_off + (r >> 6) * p.os[2] + (r & 63) * p.os[3])[i & 7] = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
    }
    const bool valid = (mask >> lane) & 1u;
    const int nv = __popc(mask), r = __popc(mask & ((1u << lane) - 1u));          // the slot's number inside the unit
    const uint32_t qb = un & 1;
    const CUtensorMap* tm = t.share ? &p.tm_k1 : &p.tm_k2;
    const uint32_t bytes = t.share ? TILE_BYTES : PAIR_BYTES;
    SlotRec rec;
    rec.flags = (r == 0 ? REC_FIRST : 0u) | (r == nv - 1 ? REC_LAST : 0u) | (t.two ? REC_TWO : 0u) | (t.share ? REC_SHARE : 0u);
    rec.w = my_w; rec.lse_off = lse_off + lane * 64; rec.out_off = out_off; rec.hk0 = t.hk0; rec.n = n; rec.chunk = my_idx; rec.unit = un; rec.pad[0] = rec.pad[1] = 0;
    ok = mbar_wait_warp(&bars[Q_EMPTY + qb], ((un >> 1) & 1) ^ 1, abort_flag, lane);
    for (int i = 0; i < nv && ok; ++i) {
#ifdef GCA_TEST_WITHHOLD_K
      // Test build only: the CTA's first K tile is never requested, so the S issuer's bounded
      // wait for it must expire.  This warp idles (bounded) until some role has given up, then
      // unwinds like after any expired wait: nothing was issued that could still be in flight
      // except the Q copy, which the drain below waits for.
      if (issued == 0) {
        if (valid && r == 0) {
          recs[0] = rec;
          mbar_arrive(&bars[REC_FULL]);
          mbar_arrive_expect_tx(&bars[Q_FULL + qb], PAIR_BYTES);
          tma_load_5d(smem + OFF_Q + qb * PAIR_BYTES, &p.tm_q, &bars[Q_FULL + qb], 0, 0, t.h0, j, n);
        }
        ++q_issued;
        for (uint32_t spin = 0; spin < 64u * GCA_WAIT_LIMIT && !*abort_flag; ++spin) __nanosleep(32);
        ok = false;
        break;
      }
#endif
      if (!(ok = mbar_wait_warp(&bars[K_EMPTY + ring.st], ring.ph ^ 1, abort_flag, lane))) break;
      if (valid && r == i) {
        if (i == 0) {
          mbar_arrive_expect_tx(&bars[Q_FULL + qb], PAIR_BYTES);
          tma_load_5d(smem + OFF_Q + qb * PAIR_BYTES, &p.tm_q, &bars[Q_FULL + qb], 0, 0, t.h0, j, n);
        }
        recs[rr.st] = rec;               // before the arrival on K_FULL: the S issuer reads it behind that barrier
        mbar_arrive(&bars[REC_FULL + rr.st]);
        mbar_arrive_expect_tx(&bars[K_FULL + ring.st], bytes);
        tma_load_5d(smem + OFF_K + ring.st * PAIR_BYTES, tm, &bars[K_FULL + ring.st], 0, 0, t.hk0, my_idx, n);
      }
      __syncwarp();
      if (i == 0) ++q_issued;
      ring.next();
      rr.next();
      ++issued;
    }
    ++un;
  }
  // end of work, in the next record of every group
  for (int i = 0; i < NWG && ok; ++i) {
    if (!(ok = mbar_wait_warp(&bars[K_EMPTY + ring.st], ring.ph ^ 1, abort_flag, lane))) break;
    if (lane == 0) {
      recs[rr.st].flags = REC_END;
      mbar_arrive(&bars[REC_FULL + rr.st]);
      if (i == 0) mbar_arrive(&bars[K_FULL + ring.st]);
    }
    ring.next();
    rr.next();
  }
  if (lane == 0 && *abort_flag) {
    drain_ring(bars, K_FULL, issued, NK);
    drain_ring(bars, Q_FULL, q_issued, 2);
  }
}

// ----------------------------------------------------------------------------- V producer
__device__ void vproducer_role(const FwdTcParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int lane) {
  if (lane != 0) return;
  const SlotRec* recs = slot_recs(smem);
  Ring ring; ring.init(NV);
  Ring rr; rr.init(NR);
  uint32_t issued = 0;
  for (;; ring.next(), rr.next(), ++issued) {
    if (!mbar_wait_bounded(&bars[REC_FULL + rr.st], rr.ph, abort_flag)) break;
    const SlotRec& rec = recs[rr.st];
    const uint32_t flags = rec.flags;
    const bool share = (flags & REC_SHARE) != 0;
    const int hk0 = rec.hk0, chunk = rec.chunk, n = rec.n;
    if (!mbar_wait_bounded(&bars[V_EMPTY + ring.st], ring.ph ^ 1, abort_flag)) break;
    if (flags & REC_END) {               // behind that wait too: the stage's previous copy may still be on its way
      mbar_arrive(&bars[V_FULL + ring.st]);
      break;
    }
    mbar_arrive_expect_tx(&bars[V_FULL + ring.st], share ? TILE_BYTES : PAIR_BYTES);
    tma_load_5d(smem + OFF_V + ring.st * PAIR_BYTES, share ? &p.tm_v1 : &p.tm_v2, &bars[V_FULL + ring.st], 0, 0, hk0, chunk, n);
  }
  if (*abort_flag) drain_ring(bars, V_FULL, issued, NV);
}

// ----------------------------------------------------------------------------- MMA issuers
// mode 0: S = Q K^T into the accumulator of group g % 3;  mode 1: O += P V with P (the slot's group's region
// of tensor memory) as the A operand.  All 32 lanes run this code; elect.sync inside the MMA /
// commit wrappers picks the issuing lane.
template <int MODE>
__device__ void issuer_role(const FwdTcParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int lane,
                            uint32_t tmem_base) {
  constexpr uint32_t PAIR16 = PAIR_BYTES >> 4, TILE16 = TILE_BYTES >> 4;
  constexpr uint32_t FULL = MODE == 0 ? K_FULL : V_FULL, EMPTY = MODE == 0 ? K_EMPTY : V_EMPTY;
  const SlotRec* recs = slot_recs(smem);
  const uint64_t dQ = umma_desc_sw128(smem_u32(smem + OFF_Q));
  const uint64_t dB = MODE == 0 ? umma_desc_sw128(smem_u32(smem + OFF_K))
                                : umma_desc_sw128_mn_blocks(smem_u32(smem + OFF_V), TILE_BYTES);
  constexpr uint32_t idesc = umma_idesc_bf16(64, 64, 0, MODE);
  Ring ring; ring.init(NK);
  Ring rr; rr.init(NR);
  uint32_t un = 0, w = 0;                     // unit; the slot's warpgroup
  for (;; ring.next(), rr.next()) {
    // tile landed and S accumulator free / P written; the record was written before that
    if (!mbar_wait_warp(&bars[FULL + ring.st], ring.ph, abort_flag, lane)) break;
    const uint32_t flags = recs[rr.st].flags;
    if (flags & REC_END) break;
    const uint32_t ub = un & 1, uph = (un >> 1) & 1;
    const uint32_t b1 = (flags & REC_SHARE) ? 0u : TILE16;             // head B's tile inside the stage
    if (flags & REC_FIRST) {
      if (!mbar_wait_warp(&bars[(MODE == 0 ? Q_FULL : O_EMPTY) + ub], MODE == 0 ? uph : uph ^ 1, abort_flag, lane)) break;
    }
    tc_fence_after();
    const uint64_t b = dB + ring.st * PAIR16;
    if (MODE == 0) {
      const uint64_t a = dQ + ub * PAIR16;
      const uint32_t dt = tmem_base + w * 64;
#pragma unroll
      for (int tl = 0; tl < 2; ++tl)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ss_elect(dt + (tl ? LANE16 : 0u), a + tl * TILE16 + kk * 2, b + (tl ? b1 : 0u) + kk * 2, idesc, (uint32_t)(kk > 0));
      umma_commit_elect(&bars[S_FULL + w]);
    } else {
      const uint32_t at = tmem_base + TMEM_P + w * 32, ot = tmem_base + TMEM_O + ub * 64, first = flags & REC_FIRST;
#pragma unroll
      for (int tl = 0; tl < 2; ++tl)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts_elect(ot + (tl ? LANE16 : 0u), at + (tl ? LANE16 : 0u) + kk * 8, b + (tl ? b1 : 0u) + kk * 128, idesc,
                             (uint32_t)(kk > 0 || !first));
      umma_commit_elect(&bars[P_EMPTY + w]);
    }
    umma_commit_elect(&bars[EMPTY + ring.st]);                          // the ring stage is free
    if (flags & REC_LAST) {
      umma_commit_elect(&bars[(MODE == 0 ? Q_EMPTY : O_FULL) + ub]);
      ++un;
    }
    if (++w == NWG) w = 0;
  }
}

// ----------------------------------------------------------------------------- softmax + epilogue
__device__ void softmax_role(const FwdTcParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int wg,
                             int quad, int lane, uint32_t tmem_base) {
  // lane 32 quad + lane of tensor memory = (head, query row) as the 64-row MMAs lay them out
  const int tile = lane >> 4;
  const int row = quad * 16 + (lane & 15);
  const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
  const bool elected = quad == 0 && lane == 0;
  const uint32_t tP = tlane + TMEM_P + (uint32_t)wg * 32, tS = tlane + (uint32_t)wg * 64;   // this warpgroup's P region and S accumulator
  const SlotRec* recs = slot_recs(smem);
  // this thread's row inside a unit's output / lse block
  __nv_bfloat16* const out_t = p.out + tile * p.os[2] + row * p.os[3];
  const long long lse_t = (long long)tile * p.K * 64 + row;
  const bool wide_store = p.wide_store != 0;
  // slots 0, 1 and 2 find their S accumulators untouched: the groups stand in for the readers of
  // "slots -3, -2 and -1" (a slot's reader arrives on the K barrier of the slot three later)
  mbar_arrive_warp(&bars[K_FULL + wg], lane);
  // The output of a unit whose last slot was this group's waits until the group has done its next slot: by then the last PV
  // product is long complete, and the other accumulator takes the next unit's products.
  bool pending = false, pend_live = false;
  __nv_bfloat16* pend_row = nullptr;
  uint32_t pend_un = 0;
  // O tile -> bf16 -> global, in four passes of ONE small loop body (16 columns: TMEM -> bf16 -> one 32-byte store per row): after
  // the first pass the body is in the instruction cache, where a straight-line conversion of all 64 columns, executed once per
  // unit, runs at instruction-fetch speed (~10 cycles per instruction measured)
  auto write_out = [&]() -> bool {
    pending = false;
    if (!mbar_wait_warp(&bars[O_FULL + (pend_un & 1)], (pend_un >> 1) & 1, abort_flag, lane)) return false;
    tc_fence_after();
    const uint32_t tO = tlane + TMEM_O + (pend_un & 1) * 64;
#pragma unroll 1
    for (int part = 0; part < 4; ++part) {
      uint32_t v[16];
      tmem_ld_32x32b_x16(tO + part * 16, v);
      tmem_ld_wait();
      if (pend_live && !GCA_DBG(4)) {
        uint32_t wv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) wv[i] = pack_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        uint8_t* dst = reinterpret_cast<uint8_t*>(pend_row) + part * 32;
        if (wide_store) st_global_256(dst, wv[0], wv[1], wv[2], wv[3], wv[4], wv[5], wv[6], wv[7]);
        else {
          reinterpret_cast<uint4*>(dst)[0] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
          reinterpret_cast<uint4*>(dst)[1] = make_uint4(wv[4], wv[5], wv[6], wv[7]);
        }
      }
    }
    tc_fence_before();
    mbar_arrive_warp(&bars[O_EMPTY + (pend_un & 1)], lane);
    return true;
  };

  uint32_t own = 0;                                 // own slots done: slot g = wg + 3 own
  uint32_t rec_st = wg, rec_ph = 0;                 // g % 18 and the parity of g / 18
  bool ok = true;
  for (;; ++own) {
    if (!(ok = mbar_wait_warp(&bars[REC_FULL + rec_st], rec_ph, abort_flag, lane))) break;
    const SlotRec& rec = recs[rec_st];
    const uint32_t flags = rec.flags;
    const uint32_t vs = (own & 1u) * NWG + wg;       // g % 6: V barrier
    if (flags & REC_END) {                           // lets the PV issuer see the end
      mbar_arrive_warp(&bars[V_FULL + vs], lane);
      break;
    }
    const float wk = rec.w;
    const long long lse_off = rec.lse_off, out_off = rec.out_off;
    const uint32_t unit = rec.unit;
    if ((rec_st += NWG) >= NR) { rec_st -= NR; rec_ph ^= 1; }
    const bool live = tile == 0 || (flags & REC_TWO);
    if (!(ok = mbar_wait_warp(&bars[S_FULL + wg], own & 1u, abort_flag, lane))) break;
    if (elected) GCA_TRACE(8, own * 3 + wg);
    tc_fence_after();
    uint32_t x[64];
    tmem_ld_32x32b_x32(tS, x);
    tmem_ld_32x32b_x32(tS + 32, x + 32);
    tmem_ld_wait();
    tc_fence_before();
    mbar_arrive_warp(&bars[K_FULL + (vs >= NWG ? vs - NWG : vs + NWG)], lane);    // the accumulator is free for slot g + 3
    if (elected) GCA_TRACE(9, own * 3 + wg);

    // row max: four independent chains of 3-input max
    float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
    if (GCA_DBG(1)) m0 = __uint_as_float(x[0]);
    else
#pragma unroll
    for (int cc = 0; cc < 64; cc += 8) {
      m0 = fmax3(m0, __uint_as_float(x[cc + 0]), __uint_as_float(x[cc + 1]));
      m1 = fmax3(m1, __uint_as_float(x[cc + 2]), __uint_as_float(x[cc + 3]));
      m2 = fmax3(m2, __uint_as_float(x[cc + 4]), __uint_as_float(x[cc + 5]));
      m3 = fmax3(m3, __uint_as_float(x[cc + 6]), __uint_as_float(x[cc + 7]));
    }
    float mm = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * p.c2;
    if (p.off_by_one > 0.f) mm = fmaxf(mm, 0.f);
    // p = exp2(x * c2 - mm): packed FMA, MUFU exp2, four packed partial sums
    const float2 c2v = make_float2(p.c2, p.c2), nmm = make_float2(-mm, -mm);
    float2 s0 = make_float2(0.f, 0.f), s1 = s0, s2 = s0, s3 = s0;
#pragma unroll
    for (int cc = 0; cc < 64; cc += 8) {
      float2 a0 = __ffma2_rn(make_float2(__uint_as_float(x[cc + 0]), __uint_as_float(x[cc + 1])), c2v, nmm);
      float2 a1 = __ffma2_rn(make_float2(__uint_as_float(x[cc + 2]), __uint_as_float(x[cc + 3])), c2v, nmm);
      float2 a2 = __ffma2_rn(make_float2(__uint_as_float(x[cc + 4]), __uint_as_float(x[cc + 5])), c2v, nmm);
      float2 a3 = __ffma2_rn(make_float2(__uint_as_float(x[cc + 6]), __uint_as_float(x[cc + 7])), c2v, nmm);
      if (!GCA_DBG(0)) {
      a0.x = ex2_approx(a0.x); a0.y = ex2_approx(a0.y);
      a1.x = ex2_approx(a1.x); a1.y = ex2_approx(a1.y);
      a2.x = ex2_approx(a2.x); a2.y = ex2_approx(a2.y);
      a3.x = ex2_approx(a3.x); a3.y = ex2_approx(a3.y);
      }
      s0 = __fadd2_rn(s0, a0); s1 = __fadd2_rn(s1, a1); s2 = __fadd2_rn(s2, a2); s3 = __fadd2_rn(s3, a3);
      x[cc + 0] = __float_as_uint(a0.x); x[cc + 1] = __float_as_uint(a0.y);
      x[cc + 2] = __float_as_uint(a1.x); x[cc + 3] = __float_as_uint(a1.y);
      x[cc + 4] = __float_as_uint(a2.x); x[cc + 5] = __float_as_uint(a2.y);
      x[cc + 6] = __float_as_uint(a3.x); x[cc + 7] = __float_as_uint(a3.y);
    }
    const float2 st2 = __fadd2_rn(__fadd2_rn(s0, s1), __fadd2_rn(s2, s3));
    float l = st2.x + st2.y;
    if (p.off_by_one > 0.f) l += p.off_by_one * ex2_approx(-mm);
    const float f = __fdividef(wk, l);
    const float2 fv = make_float2(f, f);

    if (elected) GCA_TRACE(10, own * 3 + wg);
    // PV of this group's previous slot has consumed its P
    if (own > 0 && !(ok = mbar_wait_warp(&bars[P_EMPTY + wg], (own - 1) & 1u, abort_flag, lane))) break;
    if (elected) GCA_TRACE(11, own * 3 + wg);
    // P = (w / l) * exp2(...) in bf16, two per 32-bit column, straight into tensor memory: the
    // A operand of the PV product
    uint32_t pk[32];
#pragma unroll
    for (int cc = 0; cc < 32; cc += 4) {
      const float2 q0 = __fmul2_rn(make_float2(__uint_as_float(x[2 * cc + 0]), __uint_as_float(x[2 * cc + 1])), fv);
      const float2 q1 = __fmul2_rn(make_float2(__uint_as_float(x[2 * cc + 2]), __uint_as_float(x[2 * cc + 3])), fv);
      const float2 q2 = __fmul2_rn(make_float2(__uint_as_float(x[2 * cc + 4]), __uint_as_float(x[2 * cc + 5])), fv);
      const float2 q3 = __fmul2_rn(make_float2(__uint_as_float(x[2 * cc + 6]), __uint_as_float(x[2 * cc + 7])), fv);
      pk[cc + 0] = pack_bf16x2(q0.x, q0.y); pk[cc + 1] = pack_bf16x2(q1.x, q1.y);
      pk[cc + 2] = pack_bf16x2(q2.x, q2.y); pk[cc + 3] = pack_bf16x2(q3.x, q3.y);
    }
    if (!GCA_DBG(2)) {
      tmem_st_32x32b_x32(tP, pk);
      tmem_st_wait();
    }
    tc_fence_before();
    mbar_arrive_warp(&bars[V_FULL + vs], lane);    // "P of this slot is written"
    if (elected) GCA_TRACE(12, own * 3 + wg);
    if (p.lse && live && !GCA_DBG(3)) p.lse[lse_off + lse_t] = mm + __log2f(l);
    if (pending && !(ok = write_out())) break;
    if (flags & REC_LAST) { pending = true; pend_live = live; pend_row = out_t + out_off; pend_un = unit; }
  }
  // After the last slot nothing has waited for its PV product yet; without that wait O_FULL may still be a whole unit behind, and its
  // parity would let this group through.
  if (ok && pending && mbar_wait_warp(&bars[P_EMPTY + wg], (own - 1) & 1u, abort_flag, lane)) write_out();
}

__global__ void __launch_bounds__(NTHREADS, 1)
fwd_tc_kernel(const __grid_constant__ FwdTcParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + NUM_BARS + 1);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&bars[Q_FULL + i], 1); mbar_init(&bars[Q_EMPTY + i], 1); }
    for (int i = 0; i < NWG; ++i) { mbar_init(&bars[S_FULL + i], 1); mbar_init(&bars[P_EMPTY + i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars[O_FULL + i], 1); mbar_init(&bars[O_EMPTY + i], 4); }
    for (int i = 0; i < NR; ++i) mbar_init(&bars[REC_FULL + i], 1);
    for (int i = 0; i < NK; ++i) { mbar_init(&bars[K_FULL + i], 5); mbar_init(&bars[K_EMPTY + i], 1); }   // FULL: producer + 4 warps
    for (int i = 0; i < NV; ++i) { mbar_init(&bars[V_FULL + i], 5); mbar_init(&bars[V_EMPTY + i], 1); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == SMMA_WARP) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  if (warp == KPROD_WARP && lane == 0) { tma_prefetch_desc(&p.tm_q); tma_prefetch_desc(&p.tm_k2); tma_prefetch_desc(&p.tm_k1); }
  if (warp == VPROD_WARP && lane == 0) { tma_prefetch_desc(&p.tm_v2); tma_prefetch_desc(&p.tm_v1); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  pdl_wait();

  if (warp < 4 * NWG) softmax_role(p, smem, bars, abort_flag, warp >> 2, warp & 3, lane, tmem_base);
  else if (warp == KPROD_WARP) kproducer_role(p, smem, bars, abort_flag, lane);
  else if (warp == VPROD_WARP) vproducer_role(p, smem, bars, abort_flag, lane);
  else if (warp == SMMA_WARP) issuer_role<0>(p, smem, bars, abort_flag, lane, tmem_base);
  else issuer_role<1>(p, smem, bars, abort_flag, lane, tmem_base);

  tc_fence_before();
  __syncthreads();
  if (warp == SMMA_WARP) tmem_dealloc(tmem_base, TMEM_COLS);
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicOr(p.status, GCA_STATUS_TIMEOUT);
}

long long* g_profile_buffer = nullptr;

}  // namespace

void set_fwd_profile_buffer(void* device_ptr) { g_profile_buffer = static_cast<long long*>(device_ptr); }
long long* profile_buffer() { return g_profile_buffer; }

int launch_fwd_tc(const GcaFwdArgs& a, int sms, cudaStream_t stream) {
  if (a.dtype != GCA_BF16 || a.S != 64 || a.L != 64 || a.D != 64 || a.K > 32) return GCA_ERR_ALGO;
  FwdTcParams p;
  // q viewed as (d, s, h, j, n); caches as (d, l, h, c, n).  One copy moves a 64 x 64 tile of
  // each of two consecutive heads (box extent 2 on the head axis), or of one head (tm_*1).
  int rc;
  if ((rc = make_tile_map_5d(&p.tm_q, a.q, 64, 64, a.Hq, a.J, a.N, a.q_stride[3], a.q_stride[2], a.q_stride[1], a.q_stride[0], 2))) return rc;
  if ((rc = make_tile_map_5d(&p.tm_k2, a.k_cache, 64, 64, a.Hkv, a.C, a.N, a.k_stride[2], a.k_stride[3], a.k_stride[1], a.k_stride[0], 2))) return rc;
  if ((rc = make_tile_map_5d(&p.tm_v2, a.v_cache, 64, 64, a.Hkv, a.C, a.N, a.v_stride[2], a.v_stride[3], a.v_stride[1], a.v_stride[0], 2))) return rc;
  if ((rc = make_tile_map_5d(&p.tm_k1, a.k_cache, 64, 64, a.Hkv, a.C, a.N, a.k_stride[2], a.k_stride[3], a.k_stride[1], a.k_stride[0], 1))) return rc;
  if ((rc = make_tile_map_5d(&p.tm_v1, a.v_cache, 64, 64, a.Hkv, a.C, a.N, a.v_stride[2], a.v_stride[3], a.v_stride[1], a.v_stride[0], 1))) return rc;
  p.indices = a.indices; p.weights = a.weights; p.out = (__nv_bfloat16*)a.out; p.lse = a.lse; p.status = a.status;
  for (int i = 0; i < 4; ++i) p.os[i] = a.o_stride[i];
  p.N = a.N; p.J = a.J; p.Hq = a.Hq; p.Hkv = a.Hkv; p.G = a.Hq / a.Hkv; p.K = a.K; p.C = a.C;
  p.late_first = late_chunks_first(a);
  p.pair = a.algo == GCA_ALGO_TC_UNPAIRED ? 0 : 1;
  p.dbg = 0;
#ifdef GCA_DBGKNOBS
  if (const char* dbg_env = getenv("GCA_DBG")) p.dbg = atoi(dbg_env);      // timing experiments, never in the product build
#endif
  p.HP = p.pair ? (a.Hq + 1) / 2 : a.Hq;
  const long long units = (long long)a.N * a.J * p.HP;
  if (units >= (1ll << 31) - 65536) return GCA_ERR_TOO_LARGE;
  p.units = (int)units;
  p.c2 = a.sm_scale * GCA_LOG2E;
  p.off_by_one = a.off_by_one;
  p.prof = g_profile_buffer;
  p.wide_store = (reinterpret_cast<uintptr_t>(a.out) & 31u) == 0;
  for (int i = 0; i < 4; ++i) p.wide_store = p.wide_store && (a.o_stride[i] % 16 == 0);
  if (p.units == 0) return 0;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  const unsigned grid = (unsigned)(p.units < sms ? p.units : sms);
  return (int)launch_dependent(fwd_tc_kernel, dim3(grid), dim3(NTHREADS), SMEM_BYTES, stream, p);
}

}  // namespace gca
