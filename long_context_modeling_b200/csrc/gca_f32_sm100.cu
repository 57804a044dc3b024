// GCA on float32 data with tcgen05, S = L = D = 64: every float32 operand as the sum of three bf16 values.
//
// A float32 number is b0 + b1 + b2 with b0 = bf16(x), b1 = bf16(x - b0), b2 = bf16(x - b0 - b1): three times eight bits hold its 24, exactly
// down to |x| = 2^-110, where the last of them is bf16's smallest number, 2^-133 (below, to 2^-134).  So a
// product of two float32 tiles is the sum of the bf16 products b0 b0', b0 b1', b1 b0', b1 b1', b0 b2', b2 b0' (what is left out is
// below 2^-26), accumulated from the smallest to the largest in ONE accumulator.  The tensor core cuts an accumulator off
// where an FMA rounds it, so a long chain drifts: with the large product last only its four K steps count.  Measured against
// 64 bits on N(0,1) tiles, K = 64: 7.8e-8 (2-norm), a chain of FMA 1.44e-7; the large product first: 7.5e-7.  For the same
// reason no accumulator lives longer than one retrieved chunk: O, dQ, dK and dV are summed over the chunks in registers.
//
// The A operand of (almost) every product lies in TENSOR memory, b0 of a row in lanes 0-15 of a 32-lane quarter, b1 of the same row
// 16 lanes further on: one 128-row instruction multiplies both by a piece of B, at the pipe's full rate, and the two halves of
// the accumulator belong to the same threads.  b2 has columns of its own, over zeros.  A product is 16 instructions of 128 x 64 x
// 16, 512 cycles of the tensor pipe and 256 of shared memory, against 768 and 768 as 24 instructions of 64 rows with A in
// shared memory (that form: forward 123 us, q-major 192, kv-major 220 at the size below).
//
// One CTA owns a (query chunk, head), or a (cache chunk, kv head) in the kv-major pass, and TWO CTAs share an SM: each is a
// plain chain  tiles -> scores -> workers -> second product -> workers,  and one's products run under the other's chain.
//   workers     (4 warps; 8 in the backward kernels, two groups of 32 columns each) scores -> probabilities and their
//               gradients -> three bf16 values in tensor memory; running sums in registers
//   splitters   (4 warps) fetch float32 tiles, split them and store the three bf16 tiles in the layout that the MMAs read
//   issuer      (1 warp) issues the MMAs
// The 16-row forms of tcgen05.ld / st spread a 16 x 64 tile over all 32 threads of a warp (thread t: rows t / 4 and t / 4 + 8,
// columns 2 (t % 4), + 1 of every 8), and packed pairs of what a thread holds are what the 16x128b store takes.
// Every wait is bounded (GCA_STATUS_TIMEOUT on expiry).  No atomics on results: they are bit-reproducible.
// Infinities, NaN, sums that overflow on the way and tiles of tiny numbers are outside the range of all this: such units are found by their outputs
// and done over again with multiply-adds (see `outside`), with the results that the CUDA-core kernels have always had.
// 2 x 64 chunks x 12 heads, top-8: forward 110 us, q-major 154, kv-major 200 (CUDA cores: 355, 481, 588), the whole step with inputs
// that are not in L2 520 us (1,425).  2-norm against 64 bits, N(0,1): o 2.2e-7 (4.4e-7), dq 2.8e-7 (4.7e-7), dk 3.0e-7 (6.9e-7), dv 2.6e-7
// (6.8e-7), dw 2.6e-7 (3.3e-7); the largest errors over the rms, as means over 63 drawn sizes: o 4.3e-6 (7.5e-6), dq 5.9e-6 (8.9e-6), dk 7.0e-6
// (2.0e-5), dv 6.7e-6 (1.8e-5), dw 8.6e-7 (1.1e-6), a single size now and then the other way round.  With q x 10 still closer in all five but
// dv (1.3e-6, 1.2e-6), q x 100: dq 6.7e-5 (7.6e-5), dv 1.3e-5 (6.9e-6): the kv-major pass's scores are not the forward's to the last bit.
// What bounds it now: the chains; a CTA takes ~5,400 cycles per slot in the forward, of which its own products are 1,024.
// Tried and slower: eight worker warps in the forward (the row maxima and sums then cross groups: 135 us).
#include "gca_simt.cuh"
#include "per_device.cuh"
#include "sm100_ptx.cuh"

namespace gca {

namespace {

using namespace sm100;

constexpr int PIECE = 64 * 64 * 2;                 // one bf16 tile, rows of 128 bytes, 128-byte swizzle
constexpr int TILE_BYTES = 3 * PIECE;
constexpr uint32_t PIECE16 = PIECE >> 4;
constexpr int SPLITTERS = 4, FWD_WORKERS = 4, BWD_WORKERS = 8;
constexpr int threads_of(int workers) { return (workers + SPLITTERS + 1) * 32; }
constexpr int NTILES = 4;                          // 96 KB: two CTAs per SM
constexpr int OFF_BAR = NTILES * TILE_BYTES;
constexpr int OFF_LIST = OFF_BAR + 256;            // kv-major: lse and Di of the query rows, two steps; else the slot list, Di halves
constexpr int SMEM_BYTES = OFF_LIST + 2 * 128 * 4 + 1024;
static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs per SM");
constexpr uint32_t LANE16 = 16u << 16;             // tensor-memory lanes 16-31 of every quarter
constexpr int TMEM_COLS = 256;                     // four regions of 64 columns
constexpr uint32_t R0 = 0, R1 = 64, R2 = 128, R3 = 192;
constexpr uint32_t IDESC_K = umma_idesc_bf16(128, 64, 0, 0);    // A in tensor memory, B K-major
constexpr uint32_t IDESC_MN = umma_idesc_bf16(128, 64, 0, 1);   // A in tensor memory, B MN-major
constexpr uint32_t IDESC_SS = umma_idesc_bf16(64, 64, 0, 0);    // both in shared memory, K-major
// Barriers; the meaning of the ring ones (T_*) is each kernel's own.
enum Bar { FIX_FULL = 0, A_READY = 1, T_FULL = 2, T_EMPTY = 6, S_FULL = 10, S_FREE = 11, P_FULL = 12, O_FULL = 13, O_FREE = 15, X_FULL = 16,
           DRAIN = 17, NUM_BARS = 18 };
static_assert(NUM_BARS * 8 + 8 <= 256, "barrier block");

// ---------------------------------------------------------------- tensor memory, 16-row forms
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t r[16]) {     // 32 columns
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t r[8]) {   // 16 columns of packed pairs
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

__device__ __forceinline__ float2 add2(uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1) {
  return __fadd2_rn(make_float2(__uint_as_float(a0), __uint_as_float(a1)), make_float2(__uint_as_float(b0), __uint_as_float(b1)));
}
// x, y -> the packed pair of their bf16 values; x, y keep what is left.  FIRST: a finite float32 past bf16's largest number must not become
// an infinity (an infinity ends as a NaN, which the unit's outputs show).
template <bool FIRST>
__device__ __forceinline__ uint32_t take_bf16x2(float& x, float& y) {
  uint32_t w;
  if (FIRST) asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(y), "f"(x));
  else w = pack_bf16x2(x, y);
  const float2 left = __ffma2_rn(make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), make_float2(-1.f, -1.f), make_float2(x, y));
  x = left.x;
  y = left.y;
  return w;
}

// An A operand in a region: the 32 columns of the summed axis that a group of workers holds take 16 + 16 of its 64 columns, the pair
// b0 | b1 and then b2, so that nobody writes over scores that another warp still has to read from the same region.
__device__ __forceinline__ void put_operand32(uint32_t region, int group, float v[16]) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = p == 0 ? take_bf16x2<true>(v[2 * i], v[2 * i + 1]) : p == 1 ? take_bf16x2<false>(v[2 * i], v[2 * i + 1]) : pack_bf16x2(v[2 * i], v[2 * i + 1]);
    tmem_st_16x128b_x4(region + 32 * group + (p == 1 ? LANE16 : 0u) + (p == 2 ? 16u : 0u), w);
  }
}
// The lanes below b2.  Scores in the same region write over them: then again before every use.
__device__ __forceinline__ void zero_below(uint32_t region, int group) {
  const uint32_t z[8] = {};
  tmem_st_16x128b_x4(region + 32 * group + 16 + LANE16, z);
}
// 32 columns of a 128-row product, its two halves added.
__device__ __forceinline__ void get_product32(uint32_t region, int group, float v[16]) {
  uint32_t a[16], b[16];
  tmem_ld_16x256b_x4(region + 32 * group, a);
  tmem_ld_16x256b_x4(region + 32 * group + LANE16, b);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const float2 t = add2(a[i], a[i + 1], b[i], b[i + 1]);
    v[i] = t.x;
    v[i + 1] = t.y;
  }
}
// acc += fac x the same (fac[r]: of the thread's row r)
__device__ __forceinline__ void add_product32(uint32_t region, int group, const float fac[2], float* acc) {
  float v[16];
  get_product32(region, group, v);
  const float2 f0 = make_float2(fac[0], fac[0]), f1 = make_float2(fac[1], fac[1]);
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const float2 t = __ffma2_rn((i & 2) ? f1 : f0, make_float2(v[i], v[i + 1]), make_float2(acc[i], acc[i + 1]));
    acc[i] = t.x;
    acc[i + 1] = t.y;
  }
}
// The thread's part of 32 columns of a float32 tile in global memory, and back.
__device__ __forceinline__ void load_cols32(const float* base, long long row_stride, int row, int lane, int group, float v[16]) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float* s = base + (row + 8 * r) * row_stride + 32 * group + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 t = __ldg(reinterpret_cast<const float2*>(s + 8 * i));
      v[4 * i + 2 * r] = t.x;
      v[4 * i + 2 * r + 1] = t.y;
    }
  }
}
// Returns where the thread's first value went.
__device__ __forceinline__ float* store_cols32(float* base, long long row_stride, int row, int lane, int group, const float* acc, float s) {
  base += row * row_stride + 32 * group + (lane & 3) * 2;
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(base + 8 * r * row_stride + 8 * i) = make_float2(acc[4 * i + 2 * r] * s, acc[4 * i + 2 * r + 1] * s);
  return base;
}

// ---------------------------------------------------------------- tiles
// What one of the 128 splitter threads moves of a 64 x 64 float32 tile: rows t / 8 + 16 i, columns 8 (t % 8) ... + 7.
__device__ __forceinline__ void fetch_tile(const float* src, long long row_stride, int t, float v[32]) {
  const float* s = src + (t >> 3) * row_stride + (t & 7) * 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4* r = reinterpret_cast<const float4*>(s + 16 * i * row_stride);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const float4 a = __ldg(r + x);
      v[8 * i + 4 * x] = a.x; v[8 * i + 4 * x + 1] = a.y; v[8 * i + 4 * x + 2] = a.z; v[8 * i + 4 * x + 3] = a.w;
    }
  }
}
__device__ __forceinline__ void put_tile(uint8_t* dst, float v[32], int t) {
  const int row = t >> 3;                          // row % 8 is the same for all four rows
  uint8_t* d = dst + row * 128 + (((t & 7) ^ (row & 7)) << 4);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      uint32_t w[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float &a = v[8 * i + 2 * x], &b = v[8 * i + 2 * x + 1];
        w[x] = p == 0 ? take_bf16x2<true>(a, b) : p == 1 ? take_bf16x2<false>(a, b) : pack_bf16x2(a, b);
      }
      *reinterpret_cast<uint4*>(d + i * 2048 + p * PIECE) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
// The splitters' stores are visible to the MMAs once the barrier completes (one arrival per warp).
__device__ __forceinline__ void tile_ready(uint64_t* bar, int lane) {
  fence_proxy_async_smem();
  mbar_arrive_warp(bar, lane);
}

// ---------------------------------------------------------------- products (all lanes of the issuing warp)
// D = A B with A the operand in tensor-memory region `a`: (b0 | b1) b1', (b0 | b1) b2', b2 b0', (b0 | b1) b0', in this order: the first
// writes both halves, the large one comes last.  Unrolled: an instruction is 32 cycles of the pipe, and a loop around four of them did not keep up (q-major 166 us
// against 154, kv-major 205 / 200, forward 114 / 112; around each one 202, 235, 142; as a function 187, 222, 130; with one lane elected for all 16 161, 209, 121).
template <bool MN>
__device__ __forceinline__ void product_ts(uint32_t d, uint32_t a, uint64_t b) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t aq = a + (q == 2 ? 16u : 0u);
    const uint64_t bq = b + (q == 0 ? PIECE16 : q == 1 ? 2 * PIECE16 : 0u);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      umma_bf16_ts_elect(d, aq + (kk >> 1) * 32 + (kk & 1) * 8, bq + kk * (MN ? 128 : 2), MN ? IDESC_MN : IDESC_K, (uint32_t)(q > 0 || kk > 0));
  }
}
// D = A B^T, both tiles in shared memory, K-major, 64 rows (lanes 0-15): nibble q of PA, PB is the piece.
__device__ __forceinline__ void product_ss(uint32_t d, uint64_t a, uint64_t b) {
  constexpr uint32_t PA = 0x001102u, PB = 0x010120u;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const uint64_t aq = a + ((PA >> (4 * q)) & 15u) * PIECE16, bq = b + ((PB >> (4 * q)) & 15u) * PIECE16;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) umma_bf16_ss_elect(d, aq + kk * 2, bq + kk * 2, IDESC_SS, (uint32_t)(q > 0 || kk > 0));
  }
}

// ---------------------------------------------------------------- common frame
template <int WORKERS>
struct Frame {
  static constexpr int ISSUER = WORKERS + SPLITTERS;
  uint8_t* smem;
  uint64_t* bars;
  volatile int* abort_flag;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int group = warp >> 2, row = (warp & 3) * 16 + (lane >> 2);      // group (0, 1) and first row of a worker's thread
  uint32_t tmem, quarter;          // quarter: a worker's 32 lanes of tensor memory
  __device__ __forceinline__ uint64_t k_major(int tile) const { return umma_desc_sw128(smem_u32(smem + tile * TILE_BYTES)); }
  __device__ __forceinline__ uint64_t mn_major(int tile) const { return umma_desc_sw128_mn_blocks(smem_u32(smem + tile * TILE_BYTES), PIECE); }
  __device__ __forceinline__ bool wait(int bar, uint32_t parity) const {
    return __all_sync(0xffffffffu, mbar_wait_bounded(&bars[bar], parity, abort_flag));
  }
  __device__ __forceinline__ void arrive(int bar) const { mbar_arrive_warp(&bars[bar], lane); }
  // what this worker has written to tensor memory is complete
  __device__ __forceinline__ void arrive_written(int bar) const {
    tmem_st_wait();
    tc_fence_before();
    arrive(bar);
  }
  // what this worker has read from tensor memory may be written over
  __device__ __forceinline__ void arrive_read(int bar) const {
    tc_fence_before();
    arrive(bar);
  }
  // Every CTA's operands are on their way (in registers) while its barriers and tensor memory are set up.
  __device__ __forceinline__ void set_up(uint8_t* aligned) {
    smem = aligned;
    bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
    abort_flag = reinterpret_cast<volatile int*>(slot + 1);
    if (threadIdx.x < NUM_BARS) {
      const int i = threadIdx.x;
      const bool splitters = i == FIX_FULL || (i >= T_FULL && i < T_EMPTY);
      const bool workers = i == A_READY || i == S_FREE || i == P_FULL || i == O_FREE || i == X_FULL;
      mbar_init(&bars[i], splitters ? SPLITTERS : workers ? WORKERS : 1);       // else one commit
      fence_barrier_init();
    }
    if (threadIdx.x == 0) *abort_flag = 0;
    if (warp == ISSUER) { tmem_alloc(slot, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = *slot;
    quarter = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  }
  // Whatever ended the CTA: no MMA is in flight any more when tensor memory is given back.  VOTE: true if `vote` is in some thread and no wait
  // has run out.
  template <bool VOTE = false>
  __device__ __forceinline__ bool leave(int32_t* status, bool vote = false) const {
    if (warp == ISSUER && *abort_flag) {
      umma_commit_elect(&bars[DRAIN]);
      for (int i = 0; i < (1 << 20); ++i)
        if (mbar_try_wait(&bars[DRAIN], 0)) break;
    }
    tc_fence_before();
    if (VOTE) vote = __syncthreads_or(vote);
    else __syncthreads();
    if (warp == ISSUER) tmem_dealloc(tmem, TMEM_COLS);
    if (threadIdx.x == 0 && *abort_flag && status) atomicOr(status, GCA_STATUS_TIMEOUT);
    return VOTE && vote && !*abort_flag;
  }
};
__device__ __forceinline__ uint8_t* aligned_smem(uint8_t* raw) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
}
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// The unit of a q-major CTA.  Late query chunks first: they have the most slots, and what starts last should be short.
struct UnitId {
  int n, j, h;
  __device__ __forceinline__ UnitId(const Geom& g, int b) {
    h = b % g.Hq;
    n = b / g.Hq % g.N;
    j = g.J - 1 - b / g.Hq / g.N;
  }
};
// With the list of its slots that read a chunk, x = slot, y = chunk.
struct QUnit : UnitId {
  int hk, nv;
  long long zj;
  int first;          // chunk of the first one
  unsigned valid;
  const int2* slot;
  __device__ __forceinline__ QUnit(const Geom& g, const int32_t* indices, int32_t* status, uint8_t* smem) : UnitId(g, blockIdx.x) {
    const int lane = threadIdx.x & 31;
    hk = h / g.G;
    zj = (long long)n * g.J + j;
    const int idx = lane < g.K ? slot_chunk(indices, zj, g.K, lane) : -1;
    const bool reads = idx >= 0 && idx < g.C;
    valid = __ballot_sync(0xffffffffu, reads);
    nv = __popc(valid);
    first = __shfl_sync(0xffffffffu, idx, nv ? __ffs(valid) - 1 : 0);
    int2* list = reinterpret_cast<int2*>(smem + OFF_LIST);
    if (threadIdx.x < 32) {
      if (reads) list[__popc(valid & ((1u << lane) - 1u))] = make_int2(lane, idx);
      if (status && idx >= g.C) atomicOr(status, GCA_STATUS_BAD_INDEX);
    }
    slot = list;                                   // complete behind the barrier in Frame::set_up()
  }
};

struct BwdStrides { long long dout[4], dk[4], dv[4]; };

// ------------------------------------------------------------------------------------ units outside the range
// What a warp holds of a unit's outputs lies outside the kernels' range if anything is infinite or NaN, or if nothing reaches 2^-100 (and not all
// is zero): an infinite operand or a sum past the largest number ends as a NaN here, where multiply-adds give an infinity or, for a score
// of -inf, a weight of zero; and of operands below 2^-110 bits are lost (not found: where larger ones have brought the products back above
// 2^-100, or others of the warp's outputs lie there; the split's 2^-134 of the operand, absolutely, is then the error).  The warp puts a NaN
// that no arithmetic produces in the place of its first output, and a kernel behind this one does the units so marked over again with
// multiply-adds.  Where nothing is marked the kernels behind cost 3.0 us (forward), 4.6 (q-major, which sums dw by the way; that alone took 5.2) and 3.2 (kv-major).
// HERE: the forward and the kv-major kernel do that themselves, on the spot: a launch less for short passes.  The code takes
// registers from their loops, 2.7 % of the forward and 11 % of kv-major (205 -> 228 us; q-major 165 -> 178, which has the kernel behind for dw).
constexpr unsigned MARK = 0x7fc5f32bu;
template <int N>
__device__ __forceinline__ bool outside(const float (&acc)[N]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) m = max(m, __float_as_uint(acc[i]) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  return m >= 0x7f800000u || (m > 0 && m < ((127u - 100u) << 23));
}
__device__ __forceinline__ void mark(float* first) { *reinterpret_cast<unsigned*>(first) = MARK; }
// `warps` marks, of the four row groups and (eight) the two halves of the columns
__device__ __forceinline__ bool marked(const float* tile, long long row_stride, int warps) {
  bool any = false;
  for (int w = 0; w < warps; ++w) any |= *reinterpret_cast<const volatile unsigned*>(tile + (w & 3) * 16 * row_stride + (w >> 2) * 32) == MARK;
  return any;
}
__device__ __forceinline__ int this_block() {        // looked up again rather than kept through the kernel
  int b;
  asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(b));
  return b;
}
__device__ __forceinline__ float* unit_smem() {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  return reinterpret_cast<float*>(aligned_smem(smem_raw));
}
static_assert(FWD_UNIT_SMEM <= OFF_BAR && BWD_KV_UNIT_SMEM <= OFF_BAR, "shared memory of a unit done on the spot");
// The units b, b + blocks, ...: a thread looks at one, then the block does the marked ones together.
template <class Marked, class Unit>
__device__ __forceinline__ void do_marked(int units, Marked is_marked, Unit unit) {
  pdl_wait();
  for (long long b0 = blockIdx.x; b0 < units; b0 += (long long)NTHREADS * gridDim.x) {
    const long long mine = b0 + (long long)threadIdx.x * gridDim.x;
    if (!__syncthreads_or(mine < units && is_marked((int)mine))) continue;
    for (long long b = b0; b < units && b < b0 + (long long)NTHREADS * gridDim.x; b += gridDim.x)
      if (__syncthreads_or(threadIdx.x == 0 && is_marked((int)b))) unit((int)b);
  }
}
__global__ void __launch_bounds__(NTHREADS, 4)
fwd_f32_again_kernel(const float* q, const float* kc, const float* vc, const int32_t* indices, const float* weights, float* out, float* lse, Geom g) {
  extern __shared__ __align__(16) float smem_fma[];
  do_marked(g.N * g.J * g.Hq, [&](int b) { const UnitId u(g, b); return marked(out + u.n * g.os[0] + u.j * g.os[1] + u.h * g.os[2], g.os[3], FWD_WORKERS); },
            [&](int b) { const UnitId u(g, b); fwd_unit<float>(smem_fma, u.n * g.J + u.j, u.h, q, kc, vc, indices, weights, out, lse, nullptr, g); });
}
// One block per row block: its marked heads, then dw = the sum of its heads' partials, four heads side by side, in a fixed order.
__global__ void __launch_bounds__(NTHREADS, 2)
bwd_q_f32_finish_kernel(const float* q, const float* kc, const float* vc, const int32_t* indices, const float* weights, const float* dout, const float* lse,
                        float* dq, float* dw_part, float* row_di, float* dw, Geom g, BwdStrides st) {
  extern __shared__ __align__(16) float smem_fma[];
  __shared__ float part[NTHREADS];
  const int zj = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto is_marked = [&](int h) { return h < g.Hq && marked(dq + zj / g.J * g.os[0] + zj % g.J * g.os[1] + h * g.os[2], g.os[3], BWD_WORKERS); };
  pdl_wait();
  for (int h0 = 0; h0 < g.Hq; h0 += NTHREADS) {
    if (!__syncthreads_or(is_marked(h0 + threadIdx.x))) continue;
    for (int h = h0; h < min(h0 + NTHREADS, g.Hq); ++h)
      if (__syncthreads_or(threadIdx.x == 0 && is_marked(h)))
        bwd_q_unit<float, 4>(smem_fma, zj, h, q, kc, vc, indices, weights, dout, lse, dq, dw_part, row_di, g, st.dout[0], st.dout[1], st.dout[2], st.dout[3]);
    __syncthreads();
  }
  float t = 0.f;
  if (lane < g.K)
#pragma unroll 4
    for (int h = warp; h < g.Hq; h += NTHREADS / 32) {
      const float4 v = *reinterpret_cast<const float4*>(dw_part + (((long long)zj * g.Hq + h) * g.K + lane) * 4);
      t += (v.x + v.y) + (v.z + v.w);
    }
  part[threadIdx.x] = t;
  __syncthreads();
  if (threadIdx.x < g.K) dw[(long long)zj * g.K + lane] = (part[lane] + part[32 + lane]) + (part[64 + lane] + part[96 + lane]);
}
__global__ void __launch_bounds__(NTHREADS, 2)
bwd_kv_f32_again_kernel(const float* q, const float* kc, const float* vc, const float* weights, const float* dout, const float* lse, const float* row_di,
                        float* dk, float* dv, Csr csr, Geom g, BwdStrides st) {
  extern __shared__ __align__(16) float smem_fma[];
  do_marked(g.N * g.C * g.Hkv, [&](int b) {
    const int hk = b % g.Hkv, nc = csr.unit_tab[b / g.Hkv].z;
    return marked(dk + nc / g.C * st.dk[0] + nc % g.C * st.dk[1] + hk * st.dk[3], st.dk[2], BWD_WORKERS);
  }, [&](int b) {
    bwd_kv_unit<float>(smem_fma, csr.unit_tab[b / g.Hkv], b % g.Hkv, q, kc, vc, weights, dout, lse, row_di, dk, dv, csr, g, st.dout[0], st.dout[1],
                       st.dout[2], st.dout[3], st.dk[0], st.dk[1], st.dk[2], st.dk[3], st.dv[0], st.dv[1], st.dv[2], st.dv[3]);
  });
}

// ------------------------------------------------------------------------------------ forward
// Regions: Q | scores | probabilities | product.  The next slot's scores are computed while this slot's are worked on, its product while
// the next slot's are.  The product takes exp2(S - m) / 64; w / l is a factor of the sum over the slots.
// Tiles: a ring, in the order of use K0 K1 V0 K2 V1 ...
template <bool HERE>
__global__ void __launch_bounds__(threads_of(FWD_WORKERS), 2)
fwd_f32_tc_kernel(const float* __restrict__ q, const float* __restrict__ kc, const float* __restrict__ vc,
                  const int32_t* __restrict__ indices, const float* __restrict__ weights, float* __restrict__ out,
                  float* __restrict__ lse, int32_t* status, Geom g) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const QUnit u(g, indices, status, aligned_smem(smem_raw));
  const int nv = u.nv;
  Frame<FWD_WORKERS> f;
  float v[32];
  if (nv > 0 && f.warp < FWD_WORKERS) {
#pragma unroll
    for (int h = 0; h < 2; ++h) load_cols32(q + u.n * g.qs[0] + u.j * g.qs[1] + u.h * g.qs[2], g.qs[3], f.row, f.lane, h, v + 16 * h);
  } else if (nv > 0 && f.warp < f.ISSUER)
    fetch_tile(kc + u.n * g.ks[0] + u.first * g.ks[1] + u.hk * g.ks[3], g.ks[2], threadIdx.x - FWD_WORKERS * 32, v);
  f.set_up(aligned_smem(smem_raw));
  bool again = false;

  if (f.warp < FWD_WORKERS) {
    const long long slot0 = (u.zj * g.Hq + u.h) * g.K;
    if (nv > 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        put_operand32(f.quarter + R0, h, v + 16 * h);
        zero_below(f.quarter + R0, h);
        zero_below(f.quarter + R2, h);
      }
      f.arrive_written(A_READY);
    }
    if (f.warp == 0 && lse)                        // padding slots and ids outside the cache
      for (int k = 0; k < g.K; ++k)
        if (!((u.valid >> k) & 1))
          for (int r = f.lane; r < 64; r += 32) lse[(slot0 + k) * 64 + r] = 0.f;
    const float c2 = g.sm_scale * GCA_LOG2E;
    const float w_lane = f.lane < nv ? weights[u.zj * g.K + u.slot[f.lane].x] : 0.f;
    float acc[32], p[32], fac[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int gs = 0; gs <= nv && nv > 0; ++gs) {
      float mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
      if (gs < nv) {
        if (!(ok = f.wait(S_FULL, gs & 1))) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) get_product32(f.quarter + R1, h, p + 16 * h);
        f.arrive_read(S_FREE);
#pragma unroll
        for (int i = 0; i < 32; ++i) mx[(i >> 1) & 1] = fmaxf(mx[(i >> 1) & 1], p[i]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mx[r] = quad_max(mx[r]) * c2;
          if (g.off_by_one > 0.f) mx[r] = fmaxf(mx[r], 0.f);
          mx[r] += 6.f;                            // 64 probabilities of 1 / 64: their product with V is no larger than V
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          p[i] = ex2_approx(fmaf(p[i], c2, -mx[(i >> 1) & 1]));
          l[(i >> 1) & 1] += p[i];
        }
      }
      if (gs > 0) {                                // the previous slot's product; its probabilities are no longer needed then
        if (!(ok = f.wait(O_FULL, (gs - 1) & 1))) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) add_product32(f.quarter + R3, h, fac, acc + 16 * h);
      }
      if (gs < nv) {
#pragma unroll
        for (int h = 0; h < 2; ++h) put_operand32(f.quarter + R2, h, p + 16 * h);
        f.arrive_written(P_FULL);
        const float w = __shfl_sync(0xffffffffu, w_lane, gs);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          l[r] = quad_sum(l[r]);
          if (g.off_by_one > 0.f) l[r] += g.off_by_one * ex2_approx(-mx[r]);
          fac[r] = w / l[r];
        }
        if (lse && (f.lane & 2) == 0) {            // lane % 4 = 0, 1: the thread's first and second row
          const int r = f.lane & 1;
          lse[(slot0 + u.slot[gs].x) * 64 + f.row + 8 * r] = ((r ? mx[1] : mx[0]) - 6.f) + log2f((r ? l[1] : l[0]) * 64.f);
        }
      }
    }
    if (ok) {
      float* first = nullptr;
#pragma unroll
      for (int h = 1; h >= 0; --h) first = store_cols32(out + u.n * g.os[0] + u.j * g.os[1] + u.h * g.os[2], g.os[3], f.row, f.lane, h, acc + 16 * h, 1.0f);
      again = outside(acc);
      if (!HERE && again && f.lane == 0) mark(first);
    }
  } else if (f.warp < f.ISSUER) {
    if (nv > 0) {
      const int t = threadIdx.x - FWD_WORKERS * 32;
      const float* kb = kc + u.n * g.ks[0] + u.hk * g.ks[3];
      const float* vb = vc + u.n * g.vs[0] + u.hk * g.vs[3];
      int st = 0, ph = 0;
#pragma unroll 1
      for (int i = 0; ; ++i) {
        if (!f.wait(T_EMPTY + st, ph ^ 1)) break;
        put_tile(f.smem + st * TILE_BYTES, v, t);
#ifdef GCA_TEST_WITHHOLD_K
        if (i != 1)                                // test builds: the second tile never arrives, behind scores that are under way
#endif
        tile_ready(&f.bars[T_FULL + st], f.lane);
        if (++st == NTILES) { st = 0; ph ^= 1; }
        const int y = i + 1;                       // K of slot (y + 1) / 2 and V of slot y / 2 - 1 in turn, at last V of the last slot
        if (y == 2 * nv) break;
        const bool is_k = (y & 1) && y != 2 * nv - 1;
        const int c = u.slot[y == 2 * nv - 1 ? nv - 1 : is_k ? (y + 1) / 2 : y / 2 - 1].y;
        fetch_tile(is_k ? kb + c * g.ks[1] : vb + c * g.vs[1], is_k ? g.ks[2] : g.vs[2], t, v);
      }
    }
  } else if (nv > 0 && f.wait(A_READY, 0)) {
    int st = 0, ph = 0;
#pragma unroll 1
    for (int i = 0; i < 2 * nv; ++i) {             // scores of slot 0, then scores of slot g + 1 and product of slot g in turn
      const bool product = (i & 1) == 0 ? i > 0 : i == 2 * nv - 1;
      const int gs = i == 0 ? 0 : i == 2 * nv - 1 ? nv - 1 : product ? i / 2 - 1 : (i + 1) / 2;
      if (!f.wait(T_FULL + st, ph)) break;
      if (product) {                               // the workers read the previous product before they arrived on P_FULL
        if (!f.wait(P_FULL, gs & 1)) break;
        tc_fence_after();
        product_ts<true>(f.tmem + R3, f.tmem + R2, f.mn_major(st));
      } else {
        if (gs > 0 && !f.wait(S_FREE, (gs - 1) & 1)) break;
        tc_fence_after();
        product_ts<false>(f.tmem + R1, f.tmem + R0, f.k_major(st));
      }
      umma_commit_elect(&f.bars[T_EMPTY + st]);
      umma_commit_elect(&f.bars[product ? O_FULL : S_FULL]);
      if (++st == NTILES) { st = 0; ph ^= 1; }
    }
  }
  if (f.leave<HERE>(status, again) && threadIdx.x < NTHREADS) {
    const UnitId w(g, this_block());
    fwd_unit<float>(unit_smem(), w.n * g.J + w.j, w.h, q, kc, vc, indices, weights, out, lse, nullptr, g);
  }
}

// ------------------------------------------------------------------------------------ backward, q-major
// dQ, the per-head part of dw (one partial per 16 rows), and Di = rowsum(P dP) of every (row, slot) for the kv-major pass.
// Regions: Q | dO | scores, then dS | dP, then the slot's dQ.  Tiles 0, 1: K of even and odd slots; 2, 3: V.
__global__ void __launch_bounds__(threads_of(BWD_WORKERS), 2)
bwd_q_f32_tc_kernel(const float* __restrict__ q, const float* __restrict__ kc, const float* __restrict__ vc,
                    const int32_t* __restrict__ indices, const float* __restrict__ weights, const float* __restrict__ dout,
                    const float* __restrict__ lse, float* __restrict__ dq, float* __restrict__ dw_part, float* __restrict__ row_di,
                    int32_t* status, Geom g, int beside_index, long long dos0, long long dos1, long long dos2, long long dos3) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  if (!beside_index) pdl_wait();         // else everything before the kernel that builds the index is complete: wait at the end
  const QUnit u(g, indices, nullptr, aligned_smem(smem_raw));
  const int nv = u.nv;
  Frame<BWD_WORKERS> f;
  float v[32];
  if (nv > 0 && f.warp < BWD_WORKERS) {                // group 0 brings Q, group 1 dO
    const float* src = f.group ? dout + u.n * dos0 + u.j * dos1 + u.h * dos2 : q + u.n * g.qs[0] + u.j * g.qs[1] + u.h * g.qs[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) load_cols32(src, f.group ? dos3 : g.qs[3], f.row, f.lane, h, v + 16 * h);
  } else if (nv > 0 && f.warp < f.ISSUER)
    fetch_tile(kc + u.n * g.ks[0] + u.first * g.ks[1] + u.hk * g.ks[3], g.ks[2], threadIdx.x - BWD_WORKERS * 32, v);
  f.set_up(aligned_smem(smem_raw));

  if (f.warp < BWD_WORKERS) {
    const long long slot0 = (u.zj * g.Hq + u.h) * g.K;
    if (nv > 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        put_operand32(f.quarter + (f.group ? R1 : R0), h, v + 16 * h);
        zero_below(f.quarter + (f.group ? R1 : R0), h);
      }
      f.arrive_written(A_READY);
    }
    const float w_lane = f.lane < nv ? weights[u.zj * g.K + u.slot[f.lane].x] : 0.f;
    if (f.group == 0 && f.lane < g.K && !((u.valid >> f.lane) & 1)) dw_part[(slot0 + f.lane) * 4 + f.warp] = 0.f;
    const float c2 = g.sm_scale * GCA_LOG2E, one[2] = {1.f, 1.f};
    float* part = reinterpret_cast<float*>(f.smem + OFF_LIST + 256);       // the groups' halves of Di
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int gs = 0; gs < nv; ++gs) {
      const int k = u.slot[gs].x;
      const float w = __shfl_sync(0xffffffffu, w_lane, gs);
      const float ml[2] = {lse[(slot0 + k) * 64 + f.row], lse[(slot0 + k) * 64 + f.row + 8]};
      if (!(ok = f.wait(S_FULL, gs & 1))) break;
      tc_fence_after();
      float p[16], dp[16], di[2] = {0.f, 0.f};
      get_product32(f.quarter + R2, f.group, p);
      get_product32(f.quarter + R3, f.group, dp);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int r = (i >> 1) & 1;
        p[i] = ex2_approx(fmaf(p[i], c2, -ml[r]));
        di[r] = fmaf(p[i], dp[i], di[r]);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        di[r] = quad_sum(di[r]);
        if ((f.lane & 3) == 0) part[f.group * 64 + f.row + 8 * r] = di[r];
      }
      f.arrive(X_FULL);
      if (!(ok = f.wait(X_FULL, gs & 1))) break;   // written again only behind the next scores, which need all arrivals on P_FULL
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        di[r] = part[f.row + 8 * r] + part[64 + f.row + 8 * r];
        if (f.group == 0 && (f.lane & 3) == 0) row_di[(slot0 + k) * 64 + f.row + 8 * r] = di[r];
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) p[i] = p[i] * w * (dp[i] - di[(i >> 1) & 1]);
      put_operand32(f.quarter + R2, f.group, p);
      zero_below(f.quarter + R2, f.group);
      f.arrive_written(P_FULL);
      float dsum = di[0] + di[1];                  // the 16 rows of this warp, in a fixed order
#pragma unroll
      for (int of = 16; of >= 4; of >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, of);
      if (f.group == 0 && f.lane == 0) dw_part[(slot0 + k) * 4 + f.warp] = dsum;
      if (!(ok = f.wait(O_FULL, gs & 1))) break;
      tc_fence_after();
      add_product32(f.quarter + R3, f.group, one, acc);
      f.arrive_read(O_FREE);
    }
    if (ok) {
      float* first = store_cols32(dq + u.n * g.os[0] + u.j * g.os[1] + u.h * g.os[2], g.os[3], f.row, f.lane, f.group, acc, g.sm_scale);
      if (outside(acc) && f.lane == 0) mark(first);
    }
  } else if (f.warp < f.ISSUER) {
    if (nv > 0) {
      const int t = threadIdx.x - BWD_WORKERS * 32;
      const float* kb = kc + u.n * g.ks[0] + u.hk * g.ks[3];
      const float* vb = vc + u.n * g.vs[0] + u.hk * g.vs[3];
#pragma unroll 1
      for (int i = 0; ; ++i) {                     // K and V of every slot
        const int tile = (i & 1) * 2 + ((i >> 1) & 1);
        if (!f.wait(T_EMPTY + tile, ((i >> 2) & 1) ^ 1)) break;
        put_tile(f.smem + tile * TILE_BYTES, v, t);
        tile_ready(&f.bars[T_FULL + tile], f.lane);
        if (i + 1 == 2 * nv) break;
        const bool is_k = i & 1;                   // the tile after i
        const int c = u.slot[(i + 1) >> 1].y;
        fetch_tile(is_k ? kb + c * g.ks[1] : vb + c * g.vs[1], is_k ? g.ks[2] : g.vs[2], t, v);
      }
    }
  } else if (nv > 0 && f.wait(A_READY, 0)) {
#pragma unroll 1
    for (int gs = 0; gs < nv; ++gs) {
      const int st = gs & 1, ph = (gs >> 1) & 1;
      // dS of the slot before is no longer read; then its dQ has been read
      if ((gs > 0 && !f.wait(O_FULL, (gs - 1) & 1)) || !f.wait(T_FULL + st, ph)) break;
      tc_fence_after();
      product_ts<false>(f.tmem + R2, f.tmem + R0, f.k_major(st));
      if ((gs > 0 && !f.wait(O_FREE, (gs - 1) & 1)) || !f.wait(T_FULL + 2 + st, ph)) break;
      tc_fence_after();
      product_ts<false>(f.tmem + R3, f.tmem + R1, f.k_major(2 + st));
      umma_commit_elect(&f.bars[T_EMPTY + 2 + st]);
      umma_commit_elect(&f.bars[S_FULL]);
      if (!f.wait(P_FULL, gs & 1)) break;
      tc_fence_after();
      product_ts<true>(f.tmem + R3, f.tmem + R2, f.mn_major(st));
      umma_commit_elect(&f.bars[T_EMPTY + st]);
      umma_commit_elect(&f.bars[O_FULL]);
    }
  }
  if (beside_index) pdl_wait();          // the index is complete before this kernel is
  f.leave(status);
}

// ------------------------------------------------------------------------------------ backward, kv-major
// dK, dV of one (cache chunk, kv head) over every (query chunk, slot) that retrieved it and the q heads of the group, on transposed
// scores: rows = keys, so probabilities and their gradients are the A operands of the gradient products as they stand.
// Regions: K | S^T, then w P^T | dP^T, then dS^T | dV of the step, then its dK.  Tiles 0: V; 1: dO of the step; 2, 3: Q of even and
// odd steps.  V stays in shared memory (there is no fifth region), so dP^T is the one product of 64 rows.
template <bool HERE>
__global__ void __launch_bounds__(threads_of(BWD_WORKERS), 2)
bwd_kv_f32_tc_kernel(const float* __restrict__ q, const float* __restrict__ kc, const float* __restrict__ vc,
                     const float* __restrict__ weights, const float* __restrict__ dout, const float* __restrict__ lse,
                     const float* __restrict__ row_di, float* __restrict__ dk, float* __restrict__ dv, int32_t* status, Csr csr, Geom g,
                     long long dos0, long long dos1, long long dos2, long long dos3,
                     long long dks0, long long dks1, long long dks2, long long dks3,
                     long long dvs0, long long dvs1, long long dvs2, long long dvs3) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* terms = reinterpret_cast<float*>(aligned_smem(smem_raw) + OFF_LIST);        // [step % 2]: lse | Di of the Q tile's rows
  const int hk = blockIdx.x % g.Hkv;
  const int4 unit = csr.unit_tab[blockIdx.x / g.Hkv];
  const int n = unit.z / g.C, c = unit.z % g.C;
  const int steps = (unit.y - unit.x) * g.G;       // (entry, q head of the group)
  constexpr int O_T = 1, Q_T = 2;
  auto entry_of = [&](int e) { return (int)(csr.sorted_keys[unit.x + e] & 0xffffffffull); };

  Frame<BWD_WORKERS> f;
  float v[32];
  if (steps > 0 && f.warp < BWD_WORKERS) load_cols32(kc + n * g.ks[0] + c * g.ks[1] + hk * g.ks[3], g.ks[2], f.row, f.lane, f.group, v);
  else if (steps > 0 && f.warp < f.ISSUER) fetch_tile(vc + n * g.vs[0] + c * g.vs[1] + hk * g.vs[3], g.vs[2], threadIdx.x - BWD_WORKERS * 32, v);
  f.set_up(aligned_smem(smem_raw));
  bool again = false;

  if (f.warp < BWD_WORKERS) {
    if (steps > 0) {                               // a group brings its 32 columns of K
      put_operand32(f.quarter + R0, f.group, v);
      zero_below(f.quarter + R0, f.group);
      zero_below(f.quarter + R2, f.group);         // dP^T has 64 rows: these lanes keep their zeros
      f.arrive_written(A_READY);
    }
    const float c2 = g.sm_scale * GCA_LOG2E, one[2] = {1.f, 1.f};
    float aK[16], aV[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) { aK[i] = 0.f; aV[i] = 0.f; }
    bool ok = true;
    int next = steps > 0 ? entry_of(0) : 0, sub = 0, e = 0;
#pragma unroll 1
    for (int t = 0; t < steps; ++t) {
      const float w = weights[(long long)n * g.J * g.K + next];
      if (++sub == g.G) { sub = 0; if (t + 1 < steps) next = entry_of(++e); }
      if (!(ok = f.wait(T_FULL + Q_T + (t & 1), (t >> 1) & 1) && f.wait(S_FULL, t & 1))) break;       // the terms, and the scores
      tc_fence_after();
      float p[16];
      get_product32(f.quarter + R1, f.group, p);
      uint32_t dp[16];
      tmem_ld_16x256b_x4(f.quarter + R2 + 32 * f.group, dp);
      tmem_ld_wait();
      const float* tm = terms + (t & 1) * 128 + 32 * f.group + (f.lane & 3) * 2;
      float gr[16];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 m = *reinterpret_cast<const float2*>(tm + 8 * i), d = *reinterpret_cast<const float2*>(tm + 64 + 8 * i);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int el = 4 * i + x;
          p[el] = ex2_approx(fmaf(p[el], c2, -((x & 1) ? m.y : m.x))) * w;
          gr[el] = p[el] * (__uint_as_float(dp[el]) - ((x & 1) ? d.y : d.x));
        }
      }
      put_operand32(f.quarter + R1, f.group, p);
      zero_below(f.quarter + R1, f.group);
      put_operand32(f.quarter + R2, f.group, gr);
      f.arrive_written(P_FULL);
      if (!(ok = f.wait(O_FULL, t & 1))) break;
      tc_fence_after();
      add_product32(f.quarter + R3, f.group, one, aV);
      f.arrive_read(O_FREE);
      if (!(ok = f.wait(O_FULL + 1, t & 1))) break;
      tc_fence_after();
      add_product32(f.quarter + R3, f.group, one, aK);
    }
    if (ok) {
      float* first = store_cols32(dk + n * dks0 + c * dks1 + hk * dks3, dks2, f.row, f.lane, f.group, aK, g.sm_scale);
      store_cols32(dv + n * dvs0 + c * dvs1 + hk * dvs3, dvs2, f.row, f.lane, f.group, aV, 1.0f);
      again = outside(aK) | outside(aV);
      if (!HERE && again && f.lane == 0) mark(first);
    }
  } else if (f.warp < f.ISSUER) {
    if (steps > 0) {
      const int t = threadIdx.x - BWD_WORKERS * 32;
      int entry = entry_of(0), sub = 0, e = 0;
      float term = 0.f;
#pragma unroll 1
      for (int i = 0; ; ++i) {                     // V, then Q and dO of every step s = (i - 1) / 2
        const int s = (i - 1) >> 1;
        const int tile = i == 0 ? 0 : (i & 1) ? Q_T + (s & 1) : O_T;
        if (i > 0 && !f.wait(T_EMPTY + tile, ((i & 1) ? ((s >> 1) & 1) : (s & 1)) ^ 1)) break;
        put_tile(f.smem + tile * TILE_BYTES, v, t);
        if (i & 1) terms[(s & 1) * 128 + t] = term;
        tile_ready(&f.bars[i == 0 ? FIX_FULL : T_FULL + tile], f.lane);
        if (i == 2 * steps) break;
        const int j = entry / g.K, k = entry - j * g.K, h = hk * g.G + sub;
        const bool is_q = !(i & 1);                // the tile after i
        if (is_q) {
          const long long slot = (((long long)n * g.J + j) * g.Hq + h) * g.K + k;
          term = t < 64 ? lse[slot * 64 + t] : row_di[slot * 64 + t - 64];
        }
        fetch_tile(is_q ? q + n * g.qs[0] + j * g.qs[1] + h * g.qs[2] : dout + n * dos0 + j * dos1 + h * dos2, is_q ? g.qs[3] : dos3, t, v);
        if (!is_q && ++sub == g.G) { sub = 0; if (i + 1 < 2 * steps) entry = entry_of(++e); }
      }
    }
  } else if (steps > 0 && f.wait(A_READY, 0) && f.wait(FIX_FULL, 0)) {
#pragma unroll 1
    for (int t = 0; t <= steps; ++t) {
      // S^T of step t needs P^T of the step before consumed, dP^T its dS^T; the product of 64 rows and those of 128 are kept in
      // order by waiting for their completion
      if (t > 0) {
        if (!f.wait(P_FULL, (t - 1) & 1)) break;
        tc_fence_after();
        product_ts<true>(f.tmem + R3, f.tmem + R1, f.mn_major(O_T));
        umma_commit_elect(&f.bars[T_EMPTY + O_T]);
        umma_commit_elect(&f.bars[O_FULL]);
      }
      if (t < steps) {
        if ((t > 0 && !f.wait(O_FULL, (t - 1) & 1)) || !f.wait(T_FULL + Q_T + (t & 1), (t >> 1) & 1)) break;
        tc_fence_after();
        product_ts<false>(f.tmem + R1, f.tmem + R0, f.k_major(Q_T + (t & 1)));
      }
      if (t > 0) {
        if (!f.wait(O_FREE, (t - 1) & 1)) break;
        tc_fence_after();
        product_ts<true>(f.tmem + R3, f.tmem + R2, f.mn_major(Q_T + ((t - 1) & 1)));
        umma_commit_elect(&f.bars[T_EMPTY + Q_T + ((t - 1) & 1)]);
        umma_commit_elect(&f.bars[O_FULL + 1]);
      }
      if (t < steps) {
        if ((t > 0 && !f.wait(O_FULL + 1, (t - 1) & 1)) || !f.wait(T_FULL + O_T, t & 1)) break;
        tc_fence_after();
        product_ss(f.tmem + R2, f.k_major(0), f.k_major(O_T));
        umma_commit_elect(&f.bars[S_FULL]);
      }
    }
  }
  if (f.leave<HERE>(status, again) && threadIdx.x < NTHREADS) {
    const int b = this_block();
    bwd_kv_unit<float>(unit_smem(), csr.unit_tab[b / g.Hkv], b % g.Hkv, q, kc, vc, weights, dout, lse, row_di, dk, dv, csr, g, dos0, dos1, dos2, dos3,
                       dks0, dks1, dks2, dks3, dvs0, dvs1, dvs2, dvs3);
  }
}

}  // namespace

// One CTA per unit along x: problems past that limit (no memory holds their q) stay with the CUDA-core kernels.
bool f32_tc_takes(int dtype, int S, long long units) { return dtype == GCA_F32 && S == 64 && units < (1ll << 31); }

// The kernels' shared memory, raised once per device: 0.4 us a call each, of ~90 of a small step.
static int raise_limits(int dev) {
  static PerDevice raised;
  cudaError_t rc = cudaSuccess;
  auto raise = [&](auto kernel, int bytes) {
    if (rc == cudaSuccess) rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  };
  int done = 0;
  raised.get(dev, &done, [&](int* v) {
    raise(fwd_f32_tc_kernel<false>, SMEM_BYTES);
    raise(fwd_f32_tc_kernel<true>, SMEM_BYTES);
    raise(bwd_q_f32_tc_kernel, SMEM_BYTES);
    raise(bwd_kv_f32_tc_kernel<false>, SMEM_BYTES);
    raise(bwd_kv_f32_tc_kernel<true>, SMEM_BYTES);
    raise(fwd_f32_again_kernel, FWD_UNIT_SMEM);
    raise(bwd_q_f32_finish_kernel, BWD_Q_UNIT_SMEM);
    raise(bwd_kv_f32_again_kernel, BWD_KV_UNIT_SMEM);
    *v = 1;
    return rc == cudaSuccess;
  });
  return (int)rc;
}

// As many blocks as run at once, each with a word to read for every unit it answers for: ~2 us where nothing is marked.
template <class... Params, class... Args>
static int launch_again(void (*kernel)(Params...), long long units, int blocks_per_sm, int smem, cudaStream_t stream, Args... args) {
  return (int)launch_dependent(kernel, dim3((unsigned)(units < 148 * blocks_per_sm ? units : 148 * blocks_per_sm)), dim3(NTHREADS), smem, stream, args...);
}

// (query chunk, head, slot) up to which the forward and the kv-major pass do units outside the range themselves (HERE): where the launch saved, 3 us of
// the device's time and as much of the host's, is worth the registers.  The forward at 12,096: 113.1 us against 111.5 + 3.0.  kv-major:
// steps of 40 to 936 84 us, 90 with the launch (the host's time); 1,440 and more are the device's time, 107.4 with it, 108.2 without.
constexpr long long FWD_HERE_SLOTS = 12288, KV_HERE_SLOTS = 1024;

int launch_fwd_f32_tc(const GcaFwdArgs& a, int dev, cudaStream_t stream) {
  if (int rc = raise_limits(dev)) return rc;
  const long long units = (long long)a.N * a.J * a.Hq;
  const bool here = units * a.K <= FWD_HERE_SLOTS;
  const float *q = (const float*)a.q, *kc = (const float*)a.k_cache, *vc = (const float*)a.v_cache;
  auto kernel = here ? fwd_f32_tc_kernel<true> : fwd_f32_tc_kernel<false>;
  kernel<<<(unsigned)units, threads_of(FWD_WORKERS), SMEM_BYTES, stream>>>(q, kc, vc, a.indices, a.weights, (float*)a.out, a.lse, a.status, make_geom(a));
  GCA_CUDA_CHECK(cudaGetLastError());
  if (here) return 0;
  return launch_again(fwd_f32_again_kernel, units, 4, FWD_UNIT_SMEM, stream, q, kc, vc, a.indices, a.weights, (float*)a.out, a.lse, make_geom(a));
}

int launch_bwd_f32_tc(const GcaBwdArgs& a, const Csr& csr, float* dw_part, float* row_di, int dev, cudaStream_t stream, unsigned stages) {
  if (int rc = raise_limits(dev)) return rc;
  const Geom g = make_geom(a);
  BwdStrides st;
  for (int i = 0; i < 4; ++i) { st.dout[i] = a.do_stride[i]; st.dk[i] = a.dk_stride[i]; st.dv[i] = a.dv_stride[i]; }
  const float *q = (const float*)a.q, *kc = (const float*)a.k_cache, *vc = (const float*)a.v_cache, *dout = (const float*)a.dout;
  const long long q_units = (long long)a.N * a.J * a.Hq, kv_units = (long long)a.N * a.C * a.Hkv;
  if ((stages & GCA_BWD_STAGE_Q) && q_units > 0) {
    GCA_CUDA_CHECK(launch_dependent(bwd_q_f32_tc_kernel, dim3((unsigned)q_units), dim3(threads_of(BWD_WORKERS)), SMEM_BYTES, stream, q, kc, vc,
                                    a.indices, a.weights, dout, a.lse, (float*)a.dq, dw_part, row_di, a.status, g, (int)csr.overlaps,
                                    a.do_stride[0], a.do_stride[1], a.do_stride[2], a.do_stride[3]));
    GCA_CUDA_CHECK(launch_dependent(bwd_q_f32_finish_kernel, dim3((unsigned)(a.N * a.J)), dim3(NTHREADS), BWD_Q_UNIT_SMEM, stream, q, kc, vc, a.indices,
                                    a.weights, dout, a.lse, (float*)a.dq, dw_part, row_di, (float*)a.dw, g, st));
  }
  if ((stages & GCA_BWD_STAGE_KV) && kv_units > 0) {
    const bool here = q_units * a.K <= KV_HERE_SLOTS;
    auto kernel = here ? bwd_kv_f32_tc_kernel<true> : bwd_kv_f32_tc_kernel<false>;
    kernel<<<(unsigned)kv_units, threads_of(BWD_WORKERS), SMEM_BYTES, stream>>>(
        q, kc, vc, a.weights, dout, a.lse, row_di, (float*)a.dk_cache, (float*)a.dv_cache, a.status, csr, g,
        a.do_stride[0], a.do_stride[1], a.do_stride[2], a.do_stride[3],
        a.dk_stride[0], a.dk_stride[1], a.dk_stride[2], a.dk_stride[3],
        a.dv_stride[0], a.dv_stride[1], a.dv_stride[2], a.dv_stride[3]);
    GCA_CUDA_CHECK(cudaGetLastError());
    if (here) return 0;
    return launch_again(bwd_kv_f32_again_kernel, kv_units, 2, BWD_KV_UNIT_SMEM, stream, q, kc, vc, a.weights, dout, a.lse, row_di, (float*)a.dk_cache,
                        (float*)a.dv_cache, csr, g, st);
  }
  return 0;
}

}  // namespace gca
