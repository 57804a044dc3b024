// GCA backward, q-major pass (dQ, dw and the per-row terms the kv-major pass needs) on tcgen05 /
// TMEM / TMA, bf16, S = L = D = 64.
//
// Unit = (sequence n, query chunk j, PAIR of q heads) as in the forward: Q and dO of the unit stay
// in shared memory while the K retrieved slots stream through.  Per slot the kernel recomputes
// S = Q K_k^T  and  dP = dO V_k^T;  one thread per query row forms  P = exp2(S c - LSE),
// Di = rowsum(P * dP)  (which replaces the reference's extra o = v^T p^T product,
// ltriton/gca.py:382)  and  dS = w P (dP - Di);  dQ += dS K_k  accumulates over the slots in tensor
// memory, and the per-head parts of  dw_k = sum_rows Di  go to a partials buffer that a tiny
// fixed-order kernel reduces.  For every (row, slot) the two per-row terms of the kv-major pass,
// (log2|w| - LSE) / c and -Di, are also written to the workspace, each split into three bf16
// values: the kv-major pass (gca_bwd_kv_sm100.cu), which runs AFTER this one, adds them to its
// recomputed scores with one extra MMA K step (the reference hands Di from one of its two kernels
// to the other in the same way, ltriton/gca.py:385,459).
//
// Every product is computed per head with 64-row MMAs.  A 64-row accumulator or tensor-memory
// operand occupies lanes 0-15 of every 32-lane quarter, so head B's tiles, placed at lane offset
// 16, share head A's columns: S and dP of a head PAIR take 64 columns each.  S is free again when its slot's
// worker group has read P back (~3,000 cycles after the MMAs were issued), dP when the dQ product has consumed the dS in its place
// (~4,300): three S regions, four dP regions and one dQ accumulator fill the 512 columns.
//
// A worker thread never holds a whole row in registers: it walks its 64 keys twice in passes of
// 16 columns.  Pass 1 reads S and dP, accumulates Di and writes P as packed bf16 over the S
// columns it has already read; pass 2 reads P and dP back and writes dS = P (w dP - w Di) as
// packed bf16 over the dP columns, from where the dQ product takes it as its A operand (lane =
// row of A = query row).  76 registers, which is what lets four worker groups
// and twenty-four warps fit.  Shared memory sees only the TMA copies and the MMAs' operand reads.
//
// CTA = 24 warps: four worker warpgroups, one TMA producer, three MMA issuers (S, dP, dQ), and a
// warpgroup that writes the finished dQ tiles.  The producer walks the unit list and publishes one RECORD per valid slot; the
// others follow the records and have no code that runs once per unit.  No
// atomics: gradients are bit-reproducible.  Every wait is bounded (GCA_STATUS_TIMEOUT on expiry).
//
// What bounds it (event trace at 8 x 256 chunks, 12 heads, K = 8): the S and dP issuers, ~1,280 cycles a slot inside a unit and 1,380 on
// average -- 660 and 710 of issue, 430 and 380 of waiting for tile and region -- of which the slot's 24 MMAs take 768; and close to that the regions, S 3,280
// cycles over three, dP 4,210 over four.  With three groups on three shared S / dP buffers, and every role walking the units
// by itself, it was 1,515: the groups, busy all of their 4,170 cycles a slot, and 870 cycles at each unit's end.  Each change alone gave little
// (four groups 522 -> 511 us, records with three groups 512 -> 521, separate regions with three groups 521 -> 532), together 523 -> 506,
// with one code for the S and dP issuers 500 to 507; at 1 x 1,024 chunks, K = 16 539 -> 512 to 529.
#include "gca_common.cuh"
#include "sm100_ptx.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

namespace gca {

long long* profile_buffer();

namespace {

using namespace sm100;

constexpr int TILE_BYTES = 64 * 64 * 2;
constexpr int PAIR_BYTES = 2 * TILE_BYTES;
constexpr uint32_t PAIR16 = PAIR_BYTES >> 4, TILE16 = TILE_BYTES >> 4;
// One issuing warp per product.  More were measured SLOWER, both ways tried: one warp
// per head (the heads of a slot share the region's columns) 0.835 against 0.567 ms, one warp per
// slot parity for S and dP 1,640 against 1,390 cycles per slot.
constexpr int NS = 3, NDP = 4;              // S regions, dP regions of tensor memory
constexpr int NWG = 4;                      // worker warpgroups: slot g goes to group g % 4
static_assert(NWG == NDP, "a group's dP region is its own");
constexpr int PROD_WARP = 4 * NWG, ISSUE_S = PROD_WARP + 1, ISSUE_DP = ISSUE_S + 1, ISSUE_DQ = ISSUE_DP + 1;
constexpr int WRITER_WARP = (ISSUE_DQ + 1 + 3) / 4 * 4;   // a multiple of 4: warp % 4 = its TMEM lane quarter
constexpr int NTHREADS = (WRITER_WARP + 4) * 32;
constexpr int TMEM_COLS = 512;
constexpr uint32_t LANE16 = 16u << 16;            // TMEM lane offset of head B's 64-row tile
constexpr uint32_t IDESC_64 = umma_idesc_bf16(64, 64, 0, 0);
constexpr uint32_t IDESC_DQ = umma_idesc_bf16(64, 64, 0, 1);       // A: tensor memory, B: MN-major
constexpr int STEP_K = 2;      // K-major operand: +32 bytes (>> 4) per K step of 16
constexpr int STEP_MN = 128;   // MN-major operand: +2048 bytes (>> 4) per K step of 16

constexpr int NKS = 6, NVS = 4;              // K / V ring stages
constexpr int OFF_QDO = 0;                                   // [2][Q pair | dO pair]
constexpr int OFF_K = OFF_QDO + 2 * 2 * PAIR_BYTES;          // [NKS][K pair]
constexpr int OFF_V = OFF_K + NKS * PAIR_BYTES;              // [NVS][V pair]
constexpr int OFF_BAR = OFF_V + NVS * PAIR_BYTES;
constexpr int OFF_REC = OFF_BAR + 512;                       // [NKS]
constexpr int NU = 8;                                        // unit records
constexpr int OFF_UREC = OFF_REC + NKS * 16;                 // [NU]
constexpr int SMEM_BYTES = OFF_UREC + NU * 16 + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
// A slot's record lies in the place of its K stage.  REC_FULL[stage]: it is written; K_FULL and V_FULL say so too (the same lane
// writes it and then arrives there), and who has seen PDS_FULL of the slot.  K_EMPTY of a stage -- dQ of the slot that had it is
// complete -- means that every role has read that slot's record.  UREC_FULL[u % NU]: the writer's record of unit u; when it is
// written, dP of unit u - 2 is complete, hence, with one slot a unit, dQ of unit u - 6, and the writer is past unit u - 7.
// S_FULL, DP_FULL, PDS_FULL, DP_FREE belong to a worker group, i.e. to every fourth slot.  PDS_FULL: P is read and dS written, so dQ may run
// and S of the slot three later may take the S region.
enum Bar { QDO_FULL = 0, QDO_EMPTY = 2, K_FULL = 4, K_EMPTY = K_FULL + NKS, V_FULL = K_EMPTY + NKS,
           V_EMPTY = V_FULL + NVS, S_FULL = V_EMPTY + NVS, DP_FULL = S_FULL + NWG, PDS_FULL = DP_FULL + NWG, DP_FREE = PDS_FULL + NWG,
           ACC_FULL = DP_FREE + NWG, ACC_EMPTY = ACC_FULL + 1, REC_FULL = ACC_EMPTY + 1, UREC_FULL = REC_FULL + NKS,
           NUM_BARS = UREC_FULL + NU };
static_assert(NUM_BARS * 8 + 16 <= 512, "barrier block");

// What the other roles need to know about a slot, and the writer about a unit.
struct SlotRec {
  uint32_t flags;           // REC_*
  float w;                  // retrieval weight
  long long row_off;        // element offset of (row block, head A, this slot, row 0) in lse and rowterm; 16 times that in dw_part
};
struct UnitRec {
  uint32_t flags, pad;
  long long dq_off;         // element offset of (row block, head A, row 0) in dq
};
constexpr uint32_t REC_END = 1, REC_FIRST = 2, REC_LAST = 4, REC_TWO = 8, REC_SHARE = 16;     // END: no more slots; FIRST / LAST of its unit
static_assert(sizeof(SlotRec) == 16 && sizeof(UnitRec) == 16, "records");
__device__ __forceinline__ SlotRec* slot_recs(uint8_t* smem) { return reinterpret_cast<SlotRec*>(smem + OFF_REC); }
__device__ __forceinline__ UnitRec* unit_recs(uint8_t* smem) { return reinterpret_cast<UnitRec*>(smem + OFF_UREC); }
// Tensor-memory columns: three S regions (slot g: g % 3), four dP regions (g % 4), one dQ accumulator, 64 columns each.  P (packed
// bf16, 32 columns) lands on S, dS on dP.
constexpr uint32_t COL_DP = NS * 64, COL_DQ = COL_DP + NDP * 64;
static_assert(COL_DQ + 64 <= TMEM_COLS, "tensor memory");

// x as the sum of three bf16 values (24 mantissa bits: float32 precision).
__device__ __forceinline__ void split3(float x, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(h);
  m = __float2bfloat16_rn(r1);
  l = __float2bfloat16_rn(r1 - __bfloat162float(m));
}
// The 16-byte record of one (query row, slot) for the kv-major pass: see BwdQParams::rowterm.
__device__ __forceinline__ uint4 row_terms(float a, float b) {
  __nv_bfloat16 a0, a1, a2, b0, b1, b2;
  split3(a, a0, a1, a2);
  split3(b, b0, b1, b2);
  auto pk = [](__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
  };
  return make_uint4(pk(a0, a1), pk(a2, b0), pk(b1, b2), 0u);
}
// log2|w|, kept finite: a weight of zero becomes 2^-200, which the exponential flushes to zero.
__device__ __forceinline__ float log2_abs_clamped(float w) {
  const float a = fabsf(w);
  return a > 0.f ? fmaxf(__log2f(a), -200.f) : -200.f;
}

__device__ __forceinline__ void drain(uint64_t* bars, int full0, uint32_t issued, int depth) {
  for (uint32_t back = 0; back < (uint32_t)depth && back < issued; ++back) {
    const uint32_t g = issued - 1 - back;
    for (int i = 0; i < (1 << 20); ++i)
      if (mbar_try_wait(&bars[full0 + g % depth], (g / depth) & 1)) break;
  }
}

struct BwdQParams {
  CUtensorMap tm_q, tm_do, tm_k2, tm_v2, tm_k1, tm_v1;
  int beside_index;         // launched while the index is being built (everything before THAT is complete): wait at the end, not here
  const int32_t* indices;
  const float* weights;
  const float* lse;
  __nv_bfloat16* dq;
  float* dw_part;           // (N*J, Hq, K, 4): one partial per (row block, head, slot, 16-row quarter)
  uint4* rowterm;           // (N*J, Hq, K, 64) x 16 bytes: per (row block, head, slot, query row) eight bf16 values
                            // (a0, a1, a2, b0, b1, b2, 0, 0) with a0 + a1 + a2 = (log2|w| - lse) / c2 and
                            // b0 + b1 + b2 = -Di: the kv-major pass adds them to its scores with one MMA K step
  float inv_c2;
  int32_t* status;
  Csr index;                // of a pre-gathered call, written by this kernel on its way (index.write), for the kv-major pass
  long long* prof;
  long long dqs[4];
  int units;
  int N, J, Hq, Hkv, G, K, C, HP;
  bool late_first;           // order of the units, see row_block_at
  int wide_store;           // dq rows are 32-byte aligned: 256-bit stores
  float c2, sm_scale;
};

// Heads of a unit: q heads h0, h0 + 1; their kv heads are hk0 and hk0 + 1, or both hk0 (`share`,
// grouped-query attention: one K / V tile serves both).
struct QInfo { int h0, hk0; bool two, share; };
__device__ __forceinline__ QInfo q_info(const BwdQParams& p, int hp) {
  QInfo t;
  t.h0 = 2 * hp;
  t.two = (t.h0 + 1) < p.Hq;
  if (p.G == 1) { t.hk0 = t.h0; t.share = false; }
  else { t.hk0 = t.h0 / p.G; t.share = t.two && ((t.h0 + 1) / p.G == t.hk0); }
  return t;
}
__device__ __forceinline__ int q_load_row(const BwdQParams& p, int u, int zj, int lane) {
  if (u >= p.units || lane >= p.K) return -1;
  return slot_chunk(p.indices, zj, p.K, lane);
}
__device__ __forceinline__ unsigned q_valid(const BwdQParams& p, int idx) {
  return __ballot_sync(0xffffffffu, idx >= 0 && idx < p.C);
}

// Walks this CTA's units: lane k publishes the record of slot k and issues its copies when its turn has come, the first valid lane the
// unit's record and its Q and dO copies too.  What no slot will write is also written here (rare: the first K chunks of a
// sequence): dw partials of padding slots, dQ rows of a unit without valid slots.
__device__ void q_producer(const BwdQParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int lane) {
  SlotRec* recs = slot_recs(smem);
  UnitRec* urecs = unit_recs(smem);
  PairCursor c;
  c.init(p.HP);
  Ring rk, rv; rk.init(NKS); rv.init(NVS);
  uint32_t un = 0, k_issued = 0, v_issued = 0, q_issued = 0;
  bool ok = true;
  const unsigned full = (p.K >= 32) ? 0xffffffffu : ((1u << p.K) - 1u);
  int next_zj = row_block_at(c.outer, p.N, p.J, p.late_first);
  int next_idx = q_load_row(p, c.u, next_zj, lane);
  float next_w = (c.u < p.units && lane < p.K) ? p.weights[(long long)next_zj * p.K + lane] : 0.f;
  for (; c.u < p.units && ok; c.advance()) {
    const int zj = next_zj, my_idx = next_idx;
    const float my_w = next_w;
    next_zj = row_block_at(c.next_outer(), p.N, p.J, p.late_first);
    next_idx = q_load_row(p, c.u + gridDim.x, next_zj, lane);
    next_w = (c.u + gridDim.x < p.units && lane < p.K) ? p.weights[(long long)next_zj * p.K + lane] : 0.f;
    const unsigned mask = q_valid(p, my_idx);
    const QInfo t = q_info(p, c.inner);
    const int n = zj / p.J, j = zj - n * p.J;
    const long long head_slot = ((long long)zj * p.Hq + t.h0) * p.K;                   // (row block, head A, slot 0)
    const long long dq_off = n * p.dqs[0] + j * p.dqs[1] + t.h0 * p.dqs[2];
    if (mask != full) {
      for (int i = lane; i < (t.two ? 8 : 4) * p.K; i += 32) {                              // [head][slot][quarter]
        const int x = i >> 2, k = x >= p.K ? x - p.K : x;
        if (!((mask >> k) & 1)) p.dw_part[head_slot * 4 + i] = 0.f;
      }
      if (mask == 0) {
        for (int i = lane; i < (t.two ? 128 : 64) * 8; i += 32) {
          const int r = i >> 3;
          reinterpret_cast<uint4*>(p.dq + dq_off + (r >> 6) * p.dqs[2] + (r & 63) * p.dqs[3])[i & 7] = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
    }
    const bool valid = (mask >> lane) & 1u;
    const int nv = __popc(mask), r = __popc(mask & ((1u << lane) - 1u));                    // the slot's number inside the unit
    const uint32_t ub = un & 1;
    const CUtensorMap* tmk = t.share ? &p.tm_k1 : &p.tm_k2;
    const CUtensorMap* tmv = t.share ? &p.tm_v1 : &p.tm_v2;
    const uint32_t bytes = t.share ? TILE_BYTES : PAIR_BYTES;
    const uint32_t unit_flags = (t.two ? REC_TWO : 0u) | (t.share ? REC_SHARE : 0u);
    SlotRec rec;
    rec.flags = unit_flags | (r == 0 ? REC_FIRST : 0u) | (r == nv - 1 ? REC_LAST : 0u);
    rec.w = my_w;
    rec.row_off = (head_slot + lane) * 64;
    if (!(ok = mbar_wait_warp(&bars[QDO_EMPTY + ub], ((un >> 1) & 1) ^ 1, abort_flag, lane))) break;
    for (int i = 0; i < nv; ++i) {
      const bool mine = valid && r == i;
      if (!(ok = mbar_wait_warp(&bars[K_EMPTY + rk.st], rk.ph ^ 1, abort_flag, lane))) break;
      if (mine) {
        if (i == 0) {
          UnitRec u;
          u.flags = unit_flags; u.pad = 0; u.dq_off = dq_off;
          urecs[un % NU] = u;
          mbar_arrive(&bars[UREC_FULL + un % NU]);
          uint8_t* base = smem + OFF_QDO + ub * 2 * PAIR_BYTES;
          mbar_arrive_expect_tx(&bars[QDO_FULL + ub], 2 * PAIR_BYTES);
          tma_load_5d(base, &p.tm_q, &bars[QDO_FULL + ub], 0, 0, t.h0, j, n);
          tma_load_5d(base + PAIR_BYTES, &p.tm_do, &bars[QDO_FULL + ub], 0, 0, t.h0, j, n);
        }
        recs[rk.st] = rec;               // before the arrivals on K_FULL and V_FULL: the S and dP issuers read it behind those
        mbar_arrive(&bars[REC_FULL + rk.st]);
        mbar_arrive_expect_tx(&bars[K_FULL + rk.st], bytes);
        tma_load_5d(smem + OFF_K + rk.st * PAIR_BYTES, tmk, &bars[K_FULL + rk.st], 0, 0, t.hk0, my_idx, n);
      }
      if (i == 0) ++q_issued;
      ++k_issued;
      if (!(ok = mbar_wait_warp(&bars[V_EMPTY + rv.st], rv.ph ^ 1, abort_flag, lane))) break;
      if (mine) {
        mbar_arrive_expect_tx(&bars[V_FULL + rv.st], bytes);
        tma_load_5d(smem + OFF_V + rv.st * PAIR_BYTES, tmv, &bars[V_FULL + rv.st], 0, 0, t.hk0, my_idx, n);
      }
      __syncwarp();
      ++v_issued;
      rk.next();
      rv.next();
    }
    ++un;
  }
  // end of work, in the next record of every group and of the writer (behind the waits for the stages: their last copies have landed)
  for (int i = 0; i < NWG && ok; ++i) {
    if (!(ok = mbar_wait_warp(&bars[K_EMPTY + rk.st], rk.ph ^ 1, abort_flag, lane))) break;
    if (i == 0 && !(ok = mbar_wait_warp(&bars[V_EMPTY + rv.st], rv.ph ^ 1, abort_flag, lane))) break;
    if (lane == 0) {
      recs[rk.st].flags = REC_END | (i == 0 ? REC_FIRST : 0u);
      mbar_arrive(&bars[REC_FULL + rk.st]);
      if (i == 0) {
        mbar_arrive(&bars[K_FULL + rk.st]);
        mbar_arrive(&bars[V_FULL + rv.st]);
      }
    }
    rk.next();
  }
  if (lane == 0) {
    if (ok) {
      urecs[un % NU].flags = REC_END;
      mbar_arrive(&bars[UREC_FULL + un % NU]);
    }
    if (*abort_flag) {
      drain(bars, K_FULL, k_issued, NKS);
      drain(bars, V_FULL, v_issued, NVS);
      drain(bars, QDO_FULL, q_issued, 2);
    }
  }
}

// SCORES: S per slot, or dP (dp = 1), the two warps with ONE code between them (a copy each: 507 instead of 500 us at 8 x 256 chunks, K = 8; the roles do not fit the
// instruction cache together); else dQ += dS K per slot.  All 32 lanes run this
// code; elect.sync inside the MMA / commit wrappers picks the issuing lane.  Event trace, by slot: S 0 / 1 / 2, dP 3 / 4 / 12 (before the waits, behind
// them, issued), dQ 5 / 6 (behind the waits, issued).
template <bool SCORES>
__device__ void q_issuer(uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int lane, uint32_t tmem_base, uint32_t dp, long long* prof) {
  const uint64_t dQDO = umma_desc_sw128(smem_u32(smem + OFF_QDO));
  const uint64_t dK = umma_desc_sw128(smem_u32(smem + OFF_K)), dV = umma_desc_sw128(smem_u32(smem + OFF_V));
  const uint64_t dKmn = umma_desc_sw128_mn_blocks(smem_u32(smem + OFF_K), TILE_BYTES);
  const uint32_t FULL = !SCORES ? PDS_FULL : dp ? V_FULL : K_FULL;
  const SlotRec* recs = slot_recs(smem);
  Ring rr, rv; rr.init(NKS); rv.init(NVS);                // record and K stage; V stage
  Ring rg, rf; rg.init(NWG); rf.init(NWG);                // the slot's group (and dP region); the group of slot g - 3
  uint32_t sreg = 0, un = 0, g = 0;                       // S region; unit
  bool pre_a = false, pre_b = !SCORES || !dp;                 // early probe results for the coming slot, and its flags
  uint32_t pre_flags = 0;
  for (;; ++g) {
    // S, dP: the tile has landed AND the region is free -- S: its group has read P, three slots ago; dP: dQ has consumed the
    // dS in it, four slots ago; dQ: dS is written
    const uint32_t st = !SCORES ? rg.st : dp ? rv.st : rr.st, ph = !SCORES ? rg.ph : dp ? rv.ph : rr.ph;
    if (SCORES && lane == 0) GCA_TRACE_BUF(prof, dp ? 3 : 0, g);
    if (!mbar_wait_warp2_probed(&bars[FULL + st], ph, pre_a, &bars[dp ? DP_FREE + rg.st : PDS_FULL + rf.st], dp ? rg.ph ^ 1 : rf.ph,
                                pre_b, abort_flag)) break;
    if (SCORES && g >= NS) rf.next();
    if (!pre_a) pre_flags = recs[rr.st].flags;
    const uint32_t flags = __shfl_sync(0xffffffffu, pre_flags, 0);
    if (flags & REC_END) break;
    const uint32_t ub = un & 1, uph = (un >> 1) & 1;
    const uint32_t kt1 = (flags & REC_SHARE) ? 0u : TILE16;            // head B's K / V tile inside the stage
    if (flags & REC_FIRST) {
      if (!mbar_wait_warp(&bars[SCORES ? QDO_FULL + ub : ACC_EMPTY], SCORES ? uph : ub ^ 1, abort_flag, lane)) break;
    }
    if (lane == 0) GCA_TRACE_BUF(prof, !SCORES ? 5 : dp ? 4 : 1, g);
    tc_fence_after();
    // The next slot's barriers and flags, between the two heads' MMAs: the probes' round trip runs under the issue.
    auto probe = [&] {
      Ring nr = rr, nv = rv, ng = rg;
      nr.next(); nv.next(); ng.next();
      pre_a = mbar_test_wait(&bars[FULL + (!SCORES ? ng.st : dp ? nv.st : nr.st)], !SCORES ? ng.ph : dp ? nv.ph : nr.ph);
      if (SCORES) pre_b = mbar_test_wait(&bars[dp ? DP_FREE + ng.st : PDS_FULL + rf.st], dp ? ng.ph ^ 1 : rf.ph) || (!dp && g + 1 < NS);
      if (pre_a) pre_flags = recs[nr.st].flags;
    };
    if (SCORES) {
      const uint64_t a = dQDO + ub * 2 * PAIR16 + dp * PAIR16;          // Q pair | dO pair
      const uint64_t bt = (dp ? dV : dK) + st * PAIR16;
      const uint32_t d = tmem_base + (dp ? COL_DP + rg.st * 64 : sreg);
#pragma unroll
      for (int tl = 0; tl < 2; ++tl) {
        if (tl == 1) probe();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ss_elect(d + (tl ? LANE16 : 0u), a + tl * TILE16 + kk * STEP_K, bt + (tl ? kt1 : 0u) + kk * STEP_K,
                             IDESC_64, (uint32_t)(kk > 0));
      }
      umma_commit_elect(&bars[(dp ? DP_FULL : S_FULL) + rg.st]);
      if (dp) umma_commit_elect(&bars[V_EMPTY + st]);
      if (flags & REC_LAST) umma_commit_elect(&bars[QDO_EMPTY + ub]);    // expects both issuers' commits
      if ((sreg += 64) == COL_DP) sreg = 0;
    } else {
      // dQ += dS K_k per head: A = dS from tensor memory (lane = query row, 8 columns per K step
      // of 16 keys), B = the head's K tile read N-contiguous (MN-major)
      const uint32_t acc = tmem_base + COL_DQ, at = tmem_base + COL_DP + rg.st * 64, first = flags & REC_FIRST;
      const uint64_t bk = dKmn + rr.st * PAIR16;
#pragma unroll
      for (int tl = 0; tl < 2; ++tl) {
        if (tl == 1) probe();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts_elect(acc + (tl ? LANE16 : 0u), at + (tl ? LANE16 : 0u) + kk * 8,
                             bk + (tl ? kt1 : 0u) + kk * STEP_MN, IDESC_DQ, (uint32_t)(kk > 0 || !first));
      }
      umma_commit_elect(&bars[DP_FREE + rg.st]);
      umma_commit_elect(&bars[K_EMPTY + rr.st]);        // the K tiles of this slot are free once dQ is done
      if (flags & REC_LAST) umma_commit_elect(&bars[ACC_FULL]);
    }
    if (lane == 0) GCA_TRACE_BUF(prof, !SCORES ? 6 : dp ? 12 : 2, g);
    if (flags & REC_LAST) ++un;
    rr.next();
    rv.next();
    rg.next();
  }
}

constexpr int CW = 16;                               // key columns per pass of the worker loops

// Pass 1 for 16 keys of one query row:  P = exp2(S c - LSE),  Di += P dP,  P -> packed bf16 into
// tensor memory at `dst` (8 columns of the S region that have already been read).
__device__ __forceinline__ void pass1_cols(const uint32_t* s, const uint32_t* dp, float2 c2v, float2 nl, float2& dacc, uint32_t dst) {
  uint32_t pw[CW / 2];
#pragma unroll
  for (int q = 0; q < CW; q += 2) {
    float2 a = __ffma2_rn(f2(s[q], s[q + 1]), c2v, nl);
    a.x = ex2_approx(a.x); a.y = ex2_approx(a.y);
    dacc = __ffma2_rn(a, f2(dp[q], dp[q + 1]), dacc);
    pw[q / 2] = pack_bf16x2(a.x, a.y);
  }
  tmem_st_32x32b_x8(dst, pw);
}
// Pass 2 for the same 16 keys:  dS = P (w dP - w Di)  -> packed bf16 at `dst` (8 columns of the dP
// region that have already been read).  pk: the 8 packed words of P.
__device__ __forceinline__ void pass2_cols(const uint32_t* pk, const uint32_t* dp, float2 wv, float2 nwd, uint32_t dst) {
  uint32_t ds[CW / 2];
#pragma unroll
  for (int q = 0; q < CW; q += 2) {
    const float2 pf = f2(pk[q / 2] << 16, pk[q / 2] & 0xffff0000u);
    const float2 e = __fmul2_rn(pf, __ffma2_rn(f2(dp[q], dp[q + 1]), wv, nwd));
    ds[q / 2] = pack_bf16x2(e.x, e.y);
  }
  tmem_st_32x32b_x8(dst, ds);
}
constexpr int OUT_COLS = 16, OUT_PASSES = 64 / OUT_COLS;

__device__ void q_worker(const BwdQParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int wg,
                         int quad, int lane, uint32_t tmem_base) {
  // TMEM lane of this thread = 32 quad + lane = (head tile, query row) as the 64-row MMAs lay them out
  const int tile = lane >> 4;
  const int row = quad * 16 + (lane & 15);
  const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16), td = tlane + COL_DP + wg * 64;
  const bool elected = quad == 0 && lane == 0;
  const SlotRec* recs = slot_recs(smem);
  const float2 c2v = make_float2(p.c2, p.c2);
  uint32_t st = wg, st_ph = 0, sreg = (wg % NS) * 64;             // g % 6 and the parity of g / 6; S region
  for (uint32_t own = 0;; ++own) {                               // slot g = wg + 4 own
    if (!mbar_wait_warp(&bars[REC_FULL + st], st_ph, abort_flag, lane)) break;
    const uint32_t flags = recs[st].flags;
    if (flags & REC_END) {
      // The group of the first slot behind the last lets the dQ issuer see the end: when that has seen the group's last dS (it
      // has consumed it), and the S issuer too (S of the last slot waited for it)
      if (!(flags & REC_FIRST)) break;
      const uint32_t last = wg + NWG * own - 1;
      if (own > 0 && !mbar_wait_warp(&bars[DP_FREE + wg], (own - 1) & 1u, abort_flag, lane)) break;
      if (last != ~0u && !mbar_wait_warp(&bars[S_FULL + last % NWG], (last / NWG) & 1u, abort_flag, lane)) break;
      mbar_arrive(&bars[PDS_FULL + wg]);
      break;
    }
    const float w = recs[st].w;
    const bool live = tile == 0 || (flags & REC_TWO);
    const long long block = recs[st].row_off + (tile && live ? p.K * 64 : 0);     // (row block, head, slot, row 0)
    const float lse = p.lse[block + row];
    if ((st += NWG) >= NKS) { st -= NKS; st_ph ^= 1; }
    if (!mbar_wait_warp2(&bars[S_FULL + wg], own & 1u, &bars[DP_FULL + wg], own & 1u, abort_flag, lane)) break;
    const uint32_t ts = tlane + sreg;
    if ((sreg += 64) == COL_DP) sreg = 0;                      // 4 slots on = one region on
    if (elected) GCA_TRACE_BUF(p.prof, 7, own * 4 + wg);
    tc_fence_after();
    // Pass 1 over the row's 64 keys, 16 at a time (ONE small loop body: after its first pass it
    // is in the instruction cache):  P = exp2(S c - LSE),  Di += P dP,  P -> packed bf16 over S
    // columns that earlier passes have already read.
    const float2 nl = make_float2(-lse, -lse);
    float2 dacc = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int cpos = 0; cpos < 64; cpos += CW) {
      uint32_t s[CW], dp[CW];
      tmem_ld_32x32b_x16(ts + cpos, s);
      tmem_ld_32x32b_x16(td + cpos, dp);
      tmem_ld_wait();
      pass1_cols(s, dp, c2v, nl, dacc, ts + cpos / 2);
    }
    const float di = dacc.x + dacc.y;
    tmem_st_wait();
    if (elected) GCA_TRACE_BUF(p.prof, 8, own * 4 + wg);
    // Pass 2:  dS = P (w dP - w Di)  -> packed bf16 over the dP columns already read.  (Issuing the
    // tensor-memory read of the next 16 columns before computing the current ones was measured
    // slower, 0.603 against 0.562 ms.)
    const float2 wv = make_float2(w, w), nwd = make_float2(-w * di, -w * di);
#pragma unroll 1
    for (int cpos = 0; cpos < 64; cpos += CW) {
      uint32_t pk[CW / 2], dp[CW];
      tmem_ld_32x32b_x8(ts + cpos / 2, pk);
      tmem_ld_32x32b_x16(td + cpos, dp);
      tmem_ld_wait();
      pass2_cols(pk, dp, wv, nwd, td + cpos / 2);
    }
    tmem_st_wait();
    tc_fence_before();
    mbar_arrive(&bars[PDS_FULL + wg]);
    if (elected) GCA_TRACE_BUF(p.prof, 9, own * 4 + wg);
    if (live) p.rowterm[block + row] = row_terms((log2_abs_clamped(w) - lse) * p.inv_c2, -di);
    // dw: sum of Di over the 16 rows this warp holds of each head's tile -> one partial per
    // (head, 16-row quarter)
    float dsum = di;
#pragma unroll
    for (int of = 8; of > 0; of >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, of);
    if ((lane & 15) == 0 && live) p.dw_part[block / 16 + quad] = dsum;
  }
}

// The dQ writer: a warpgroup of its own, so that no worker group is held up by a unit's output (a
// worker group is tied to every fourth slot; while it waited for the unit's last dQ product and
// stored the tile, ~2,000-2,800 cycles, its next slot and with it the whole ring stood still once
// per unit: 0.571 -> 0.544 ms).  Its wait is the ordinary suspending try_wait: polling with a sleep
// between probes (20 / 100 / 400 ns) was measured slower (0.584 / 0.574 / 0.558 ms).  Thread = TMEM
// lane = (head tile, query row) as in the workers.
__device__ void q_writer(const BwdQParams& p, uint8_t* smem, uint64_t* bars, volatile int* abort_flag, int quad, int lane, uint32_t tmem_base) {
  const int tile = lane >> 4;
  const int row = quad * 16 + (lane & 15);
  const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
  const bool elected = quad == 0 && lane == 0;
  const UnitRec* urecs = unit_recs(smem);
  __nv_bfloat16* const dq_t = p.dq + tile * p.dqs[2] + row * p.dqs[3];
  for (uint32_t un = 0;; ++un) {
    if (!mbar_wait_warp(&bars[UREC_FULL + un % NU], (un / NU) & 1, abort_flag, lane)) break;
    const uint32_t flags = urecs[un % NU].flags;
    if (flags & REC_END) break;
    const bool live = tile == 0 || (flags & REC_TWO);
    __nv_bfloat16* dq_row = dq_t + urecs[un % NU].dq_off;
    if (!mbar_wait_warp(&bars[ACC_FULL], un & 1, abort_flag, lane)) break;
    if (elected) GCA_TRACE_BUF(p.prof, 10, un);
    tc_fence_after();
    // the whole row into registers, so that the accumulator is free again at once
    uint32_t v[64];
    tmem_ld_32x32b_x32(tlane + COL_DQ, v);
    tmem_ld_32x32b_x32(tlane + COL_DQ + 32, v + 32);
    tmem_ld_wait();
    tc_fence_before();
    mbar_arrive_warp(&bars[ACC_EMPTY], lane);
#pragma unroll
    for (int part = 0; part < OUT_PASSES; ++part)
      if (live) store16_bf16(reinterpret_cast<uint8_t*>(dq_row) + part * OUT_COLS * 2, v + part * OUT_COLS, p.sm_scale, p.wide_store);
    if (elected) GCA_TRACE_BUF(p.prof, 11, un);
  }
}

__global__ void __launch_bounds__(NTHREADS, 1)
bwd_q_tc_kernel(const __grid_constant__ BwdQParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + NUM_BARS + 1);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars[QDO_FULL + i], 1);
      mbar_init(&bars[QDO_EMPTY + i], 2);                  // S issuers + dP issuers
    }
    mbar_init(&bars[ACC_FULL], 1);
    mbar_init(&bars[ACC_EMPTY], 4);
    for (int i = 0; i < NWG; ++i) {
      mbar_init(&bars[S_FULL + i], 1); mbar_init(&bars[DP_FULL + i], 1); mbar_init(&bars[PDS_FULL + i], 128); mbar_init(&bars[DP_FREE + i], 1);
    }
    for (int i = 0; i < NKS; ++i) { mbar_init(&bars[K_FULL + i], 1); mbar_init(&bars[K_EMPTY + i], 1); mbar_init(&bars[REC_FULL + i], 1); }
    for (int i = 0; i < NU; ++i) mbar_init(&bars[UREC_FULL + i], 1);
    for (int i = 0; i < NVS; ++i) { mbar_init(&bars[V_FULL + i], 1); mbar_init(&bars[V_EMPTY + i], 1); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == ISSUE_S) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  if (warp == PROD_WARP && lane == 0) {
    tma_prefetch_desc(&p.tm_q); tma_prefetch_desc(&p.tm_do); tma_prefetch_desc(&p.tm_k2); tma_prefetch_desc(&p.tm_v2);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  if (!p.beside_index) pdl_wait();
  if (warp < 4 * NWG) q_worker(p, smem, bars, abort_flag, warp >> 2, warp & 3, lane, tmem_base);
  else if (warp == PROD_WARP) q_producer(p, smem, bars, abort_flag, lane);
  else if (warp >= WRITER_WARP) q_writer(p, smem, bars, abort_flag, warp & 3, lane, tmem_base);
  else if (warp == ISSUE_S || warp == ISSUE_DP) q_issuer<true>(smem, bars, abort_flag, lane, tmem_base, (uint32_t)(warp - ISSUE_S), p.prof);
  else if (warp == ISSUE_DQ) q_issuer<false>(smem, bars, abort_flag, lane, tmem_base, 0u, p.prof);
  if (p.beside_index) pdl_wait();        // the index is complete before this kernel is
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUE_S) tmem_dealloc(tmem_base, TMEM_COLS);
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicOr(p.status, GCA_STATUS_TIMEOUT);
  if (p.index.write) {
    for (int i = (int)(blockIdx.x * NTHREADS + threadIdx.x); i < p.N * p.C; i += (int)gridDim.x * NTHREADS) identity_entry(p.index, i, p.C);
  }
}

// every 64-element bf16 row of the tensor starts on a 32-byte boundary
bool rows_32b_aligned(const void* base, const int64_t* stride) {
  if (reinterpret_cast<uintptr_t>(base) & 31u) return false;
  for (int i = 0; i < 4; ++i)
    if (stride[i] % 16 != 0) return false;
  return true;
}

}  // namespace

// dw_part: (N*J, Hq, K, 4) float32 partials; rowterm: (N*J, Hq, K, 64) x 16 bytes (see BwdQParams).
int launch_bwd_q_tc(const GcaBwdArgs& a, float* dw_part, uint4* rowterm, const Csr& csr, int sms, cudaStream_t stream) {
  const float c2 = a.sm_scale * GCA_LOG2E;
  int rc;
  auto qmap = [&](CUtensorMap* m, const void* base, const int64_t* st, int box) {
    return make_tile_map_5d(m, base, 64, 64, a.Hq, a.J, a.N, st[3], st[2], st[1], st[0], box);
  };
  auto kmap = [&](CUtensorMap* m, const void* base, const int64_t* st, int box) {
    return make_tile_map_5d(m, base, 64, 64, a.Hkv, a.C, a.N, st[2], st[3], st[1], st[0], box);
  };
  BwdQParams p;
  p.index = csr;
  if ((rc = qmap(&p.tm_q, a.q, a.q_stride, 2)) || (rc = qmap(&p.tm_do, a.dout, a.do_stride, 2)) ||
      (rc = kmap(&p.tm_k2, a.k_cache, a.k_stride, 2)) || (rc = kmap(&p.tm_v2, a.v_cache, a.v_stride, 2)) ||
      (rc = kmap(&p.tm_k1, a.k_cache, a.k_stride, 1)) || (rc = kmap(&p.tm_v1, a.v_cache, a.v_stride, 1)))
    return rc;
  p.indices = a.indices; p.weights = a.weights; p.lse = a.lse;
  p.dq = (__nv_bfloat16*)a.dq; p.dw_part = dw_part; p.rowterm = rowterm; p.inv_c2 = 1.0f / c2; p.status = a.status;
  p.prof = profile_buffer();
  for (int i = 0; i < 4; ++i) p.dqs[i] = a.dq_stride[i];
  p.N = a.N; p.J = a.J; p.Hq = a.Hq; p.Hkv = a.Hkv; p.G = a.Hq / a.Hkv; p.K = a.K; p.C = a.C;
  p.HP = (a.Hq + 1) / 2;
  const long long units = (long long)a.N * a.J * p.HP;
  if (units >= (1ll << 31) - 65536) return GCA_ERR_TOO_LARGE;
  p.units = (int)units;
  p.late_first = late_chunks_first(a);
  p.c2 = c2; p.sm_scale = a.sm_scale;
  p.wide_store = rows_32b_aligned(a.dq, a.dq_stride);
  if (p.units == 0) return 0;
  GCA_CUDA_CHECK(cudaFuncSetAttribute(bwd_q_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  const unsigned grid = (unsigned)(p.units < sms ? p.units : sms);
  p.beside_index = csr.overlaps;
  return (int)launch_dependent(bwd_q_tc_kernel, dim3(grid), dim3(NTHREADS), SMEM_BYTES, stream, p);
}

}  // namespace gca
