// Attention of one or two query rows over rows of a bf16 cache, sixteen keys at a time in one warp, several sixteens in a row.  The bound
// is HBM, but with a multiply-add per value the instructions were in the way of the loads: 384 items x 512 keys were 6.6 million warp
// instructions, as matrix instructions (m16n8k16, float32 sums) they are 3.9 million, most of them for the softmax and around the keys.
//
// Lane = 4 * g + t.  Scores: the keys are the rows of A.  A lane's 16 bytes of a key row are the four registers of one A operand, as
// they come from memory: its dims 0,1 and 4,5 stand in row g, dims 2,3 and 6,7 in row g + 8.  So the columns of B come in pairs, the
// query at the dims of the one and of the other, and the score is D[g][2c] + D[g + 8][2c + 1].  Two operands are a key's 64 dims.
// Outputs: the dims are the rows of A (a permute of two keys' values makes its registers), the keys the contraction, and
// every weight stands in three columns as the sum of three bf16 values, which is all of its 24 bits: nothing is rounded to 16.
#pragma once
#include "gca_common.cuh"

namespace gca {
namespace row_attn {

__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float finite_max(float m) { return m == -INFINITY ? 0.f : m; }       // nothing seen yet: ex2(-inf - 0) = 0
__device__ __forceinline__ uint32_t pack(float a, float b) {                                      // a in the low half
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float low(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ uint4 load16(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }

// The query rows as B: registers [dims 0-31, 32-63][low, high half of the contraction].  row0, row1: the lane's 8 t .. of the rows.
struct Query { uint32_t b[2][2]; };
template <int R>
__device__ __forceinline__ Query query(const __nv_bfloat16* row0, const __nv_bfloat16* row1, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const __nv_bfloat16* row = R == 2 && (g & 2) ? row1 : row0;
  Query q;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    uint4 w = make_uint4(0, 0, 0, 0);
    if (row) w = load16(row + u * 32 + t * 8);
    q.b[u][0] = g & 1 ? w.y : w.x; q.b[u][1] = g & 1 ? w.w : w.z;
  }
  return q;
}

// Sixteen keys: the lane holds [key g, key 8 + g][dims 8 t .., 32 + 8 t ..] of K and dims 8 g .. of the keys 2t, 2t + 1, 8 + 2t, 9 + 2t of V.
__device__ __forceinline__ int key_of_k(int lane, int h) { return h * 8 + (lane >> 2); }
__device__ __forceinline__ int key_of_v(int lane, int s) { return (s >> 1) * 8 + (lane & 3) * 2 + (s & 1); }

// Running state.  m, l: of the row `lane & 1` (R = 2); l is this lane's part, of keys g and 8 + g.  acc[i]: dims 8 g + 2 i (0, 1) and 8 g + 2 i + 1
// (2, 3) of the columns 2 t, 2 t + 1.
struct State { float m, l, acc[4][4]; };
__device__ __forceinline__ void reset(State& st) {
  st.m = -INFINITY; st.l = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) st.acc[i][c] = 0.f;
}

// Dot products of the keys g and 8 + g with the row `lane & 1` (R = 2).
__device__ __forceinline__ void scores(const Query& q, const uint4 (&k)[2][2], float (&s)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 2; ++u) mma(d, k[h][u].x, k[h][u].y, k[h][u].z, k[h][u].w, q.b[u][0], q.b[u][1]);
    s[h] = d[0] + d[3];
  }
}

// s: the scores in log2 units, -inf where masked (the values of a masked key are finite).
template <int R>
__device__ __forceinline__ void accumulate(State& st, float (&s)[2], const uint4 (&v)[4], int lane) {
  const int g = lane >> 2, t = lane & 3;
  float m = fmaxf(st.m, fmaxf(s[0], s[1]));
#pragma unroll
  for (int of = 4; of < 32; of <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, of));
  const float mf = finite_max(m), corr = ex2(st.m - mf);
  st.m = m;
  const float p0 = ex2(s[0] - mf), p1 = ex2(s[1] - mf);
  st.l = fmaf(st.l, corr, p0 + p1);
  // the three parts of both weights, keys g and 8 + g in one register
  const uint32_t w1 = pack(p0, p1);
  const float r0 = p0 - low(w1), r1 = p1 - high(w1);
  const uint32_t w2 = pack(r0, r1), w3 = pack(r0 - low(w2), r1 - high(w2));
  uint32_t x, y;                                                 // of keys 2t (and 8 + 2t), 2t + 1 (and 9 + 2t): column g's part
  if (R == 1) {                                                  // column = part; lane t of a key offers part t
    const uint32_t w = t == 0 ? w1 : t == 1 ? w2 : t == 2 ? w3 : 0u;
    const int src = t * 8 + min(g, 3);
    x = __shfl_sync(0xffffffffu, w, src); y = __shfl_sync(0xffffffffu, w, src + 4);
  } else {                                                       // column = 2 * part + row; lane t offers parts 0, 1 of row t & 1, and part 2
    const uint32_t w = t < 2 ? w1 : w2;
    const int src = t * 8 + (g & 3), last = t * 8 + (g & 1);
    x = __shfl_sync(0xffffffffu, w, src); y = __shfl_sync(0xffffffffu, w, src + 4);
    const uint32_t x3 = __shfl_sync(0xffffffffu, w3, last), y3 = __shfl_sync(0xffffffffu, w3, last + 4);
    if (g >= 4) { x = g < 6 ? x3 : 0u; y = g < 6 ? y3 : 0u; }
  }
  const uint32_t b0 = __byte_perm(x, y, 0x5410), b1 = __byte_perm(x, y, 0x7632);
  float c0 = corr, c1 = corr;
  if (R == 2) {
    const float other = __shfl_xor_sync(0xffffffffu, corr, 1);
    c0 = t & 1 ? other : corr; c1 = t & 1 ? corr : other;
  }
  const float2 c2 = make_float2(c0, c1);
  const uint32_t vw[4][4] = {{v[0].x, v[0].y, v[0].z, v[0].w}, {v[1].x, v[1].y, v[1].z, v[1].w}, {v[2].x, v[2].y, v[2].z, v[2].w}, {v[3].x, v[3].y, v[3].z, v[3].w}};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 lo2 = __fmul2_rn(make_float2(st.acc[i][0], st.acc[i][1]), c2), hi2 = __fmul2_rn(make_float2(st.acc[i][2], st.acc[i][3]), c2);
    st.acc[i][0] = lo2.x; st.acc[i][1] = lo2.y; st.acc[i][2] = hi2.x; st.acc[i][3] = hi2.y;
    mma(st.acc[i], __byte_perm(vw[0][i], vw[1][i], 0x5410), __byte_perm(vw[0][i], vw[1][i], 0x7632), __byte_perm(vw[2][i], vw[3][i], 0x5410),
        __byte_perm(vw[2][i], vw[3][i], 0x7632), b0, b1);
  }
}

// The warp's state as a whole: sums l over its lanes (of row `lane & 1`) and the parts: out[r][e] is dim 8 g + e of row r, in the lanes t = 0.
// An infinite value leaves the parts inf and NaN (0 x inf): the first part alone then is the product.
template <int R>
__device__ __forceinline__ void finish(State& st, float (&out)[R][8]) {
#pragma unroll
  for (int of = 4; of < 32; of <<= 1) st.l += __shfl_xor_sync(0xffffffffu, st.l, of);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float a = st.acc[i][2 * e], b = st.acc[i][2 * e + 1];
      if (R == 1) {
        const float sum = a + (b + __shfl_down_sync(0xffffffffu, a, 1));
        out[0][2 * i + e] = sum != sum ? a : sum;
      } else {
        const float s0 = a + (__shfl_down_sync(0xffffffffu, a, 1) + __shfl_down_sync(0xffffffffu, a, 2));
        const float s1 = b + (__shfl_down_sync(0xffffffffu, b, 1) + __shfl_down_sync(0xffffffffu, b, 2));
        out[0][2 * i + e] = s0 != s0 ? a : s0; out[R - 1][2 * i + e] = s1 != s1 ? b : s1;
      }
    }
}

}  // namespace row_attn
}  // namespace gca
