// Shared declarations for the GCA kernels: argument views, dtype helpers, error checks.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gca_b200.h"

#define GCA_LOG2E 1.4426950408889634f

#define GCA_CUDA_CHECK(expr)                         \
  do {                                               \
    cudaError_t _e = (expr);                         \
    if (_e != cudaSuccess) return (int)_e;           \
  } while (0)

namespace gca {

// Element-typed load/store that always computes in float.
template <typename T> __device__ __forceinline__ float ld_f(const T* p);
template <> __device__ __forceinline__ float ld_f<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ld_f<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <typename T> __device__ __forceinline__ void st_f(T* p, float v);
template <> __device__ __forceinline__ void st_f<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void st_f<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

// The chunk that slot k of query chunk zj reads; no index array = the pre-gathered call, slot k reads chunk k.
__device__ __forceinline__ int slot_chunk(const int32_t* __restrict__ indices, long long zj, int K, int k) {
  return indices ? indices[zj * K + k] : k;
}

// Programmatic dependent launch: a kernel launched with `launch_dependent` may start while the one before it on the
// stream still runs (once every block of that one has called pdl_trigger or left); pdl_wait returns when
// everything before it on the stream is complete and visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... Params, class... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// The same as pairs of CTAs (clusters of two along x).
template <class... Params, class... Args>
inline cudaError_t launch_dependent_pairs(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// Problem geometry shared by forward and backward kernels (passed by value).
struct Geom {
  int N, J, Hq, Hkv, S, L, D, K, C, G;
  long long qs[4];   // q   strides n, j, h, s
  long long os[4];   // out / dq strides
  long long ks[4];   // k   strides n, c, l, h
  long long vs[4];   // v   strides n, c, l, h
  float sm_scale;
  float off_by_one;
};

inline Geom make_geom(const GcaFwdArgs& a) {
  Geom g;
  g.N = a.N; g.J = a.J; g.Hq = a.Hq; g.Hkv = a.Hkv; g.S = a.S; g.L = a.L; g.D = a.D; g.K = a.K; g.C = a.C;
  g.G = a.Hq / a.Hkv;
  for (int i = 0; i < 4; ++i) { g.qs[i] = a.q_stride[i]; g.os[i] = a.o_stride[i]; g.ks[i] = a.k_stride[i]; g.vs[i] = a.v_stride[i]; }
  g.sm_scale = a.sm_scale; g.off_by_one = a.off_by_one;
  return g;
}

inline Geom make_geom(const GcaBwdArgs& a) {
  Geom g;
  g.N = a.N; g.J = a.J; g.Hq = a.Hq; g.Hkv = a.Hkv; g.S = a.S; g.L = a.L; g.D = a.D; g.K = a.K; g.C = a.C;
  g.G = a.Hq / a.Hkv;
  for (int i = 0; i < 4; ++i) { g.qs[i] = a.q_stride[i]; g.os[i] = a.dq_stride[i]; g.ks[i] = a.k_stride[i]; g.vs[i] = a.v_stride[i]; }
  g.sm_scale = a.sm_scale; g.off_by_one = a.off_by_one;
  return g;
}

// Inverse retrieval index: for every cache chunk (n, c) the list of (j*K + k) entries that retrieved it, in order: the low
// 32 bits of `sorted_keys`.
// `unit_tab` lists the chunks in the order the kv-major kernels take them: by DECREASING number of
// retrievers, sequence by sequence or of all sequences (units_by_count); x = first entry,
// y = one past the last, z = chunk id n*C + c.
// `tickets`: two counters, zero between launches: units handed out by the tensor-core kv-major kernel, CTAs that are done.
// `overlaps`: the kernel that builds it was just launched and lets the next kernel on the stream start before it is done.
struct Csr {
  const unsigned long long* sorted_keys;
  const int4* unit_tab;
  int* tickets;
  bool overlaps;
  bool write = false;      // laid out only: the q-major pass writes it
};

// The index of a pre-gathered call: chunk c of row block n is read by its slot c and nothing else.
__device__ __forceinline__ void identity_entry(const Csr& index, int i, int C) {
  const_cast<unsigned long long*>(index.sorted_keys)[i] = ((unsigned long long)i << 32) | (unsigned)(i % C);
  const_cast<int4*>(index.unit_tab)[i] = make_int4(i, i + 1, i, 0);
  if (i < 2) index.tickets[i] = 0;
}

// launch == false: only lay the index out in `workspace` (it was built by an earlier call)
// by_count: the unit table's order (units_by_count)
// by_sort: take the radix-sort path even where the single-launch path would do (same bits)
int build_csr(const int32_t* indices, int N, int J, int K, int C, void* workspace, size_t workspace_bytes,
              bool by_count, Csr* out, size_t* used_bytes, cudaStream_t stream, bool launch = true, bool by_sort = false);
size_t csr_workspace_bytes(int N, int J, int K, int C);

// SIMT (CUDA-core, fp32 accumulate) kernels: every dtype, S <= 64, L = D = 64.
int launch_fwd_simt(const GcaFwdArgs& a, cudaStream_t stream);
// stages: GCA_BWD_STAGE_KV and / or GCA_BWD_STAGE_Q
// row_di: (N*J, Hq, K, 64) floats of scratch, Di of every row: the q-major stage writes it, the kv-major stage reads it
int launch_bwd_simt(const GcaBwdArgs& a, const Csr& csr, float* dw_part, float* row_di, cudaStream_t stream, unsigned stages);

// float32 on the tensor cores, S = L = D = 64 (same scratch; four dw partials per (row block, head, slot), summed to dw by the q-major stage).
bool f32_tc_takes(int dtype, int S, long long units);
int launch_fwd_f32_tc(const GcaFwdArgs& a, int dev, cudaStream_t stream);
int launch_bwd_f32_tc(const GcaBwdArgs& a, const Csr& csr, float* dw_part, float* row_di, int dev, cudaStream_t stream, unsigned stages);

// tcgen05 / TMEM / TMA kernels: bf16, S = L = D = 64.
int launch_fwd_tc(const GcaFwdArgs& a, int sms, cudaStream_t stream);
// rowterm: (N*J, Hq, K, 64) x 16 bytes of scratch the q-major pass fills with the per-row terms of the kv-major pass
int launch_bwd_tc(const GcaBwdArgs& a, const Csr& csr, float* dw_part, uint4* rowterm, int sms, cudaStream_t stream, unsigned stages);

// dw[zj, k] = sum over heads and `parts` partials of dw_part[zj, h, k, part], in a fixed order
int launch_dw_reduce(const float* dw_part, float* dw, int ZJ, int Hq, int K, int parts, cudaStream_t stream);
int bwd_tc_dw_parts();   // partials per (row block, head, slot) that the tensor-core q-major pass writes

// Order of the kv-major kernels' units, the rows of the unit table.  A chunk near the start of a sequence has many times the retrievers of one near its end, so
// the large units have to start first; over ALL sequences when what they read, Q and dO, stays in L2 whatever the order
// (half of its 126 MB), else one sequence after the other, which reads each sequence's Q and dO from memory once.
inline bool units_by_count(const GcaBwdArgs& a) {
  return (long long)a.N * a.J * a.Hq * a.S * a.D * 2 * (a.dtype == GCA_F32 ? 4 : 2) <= (64ll << 20);
}

// Order of the forward's and the q-major pass's units.  The first query chunks of a sequence have few or no chunks behind them to
// retrieve: taken last, these short units even the CTAs out, where a last, partial wave in ascending order is made of the longest.  That pays
// where a CTA has few units (3 x 37 chunks, 12 heads, K = 8, 4.4 units a CTA: the forward's kernel 34.9 -> 32.4 us).  Side by
// side the sequences have to share L2, hence the line at half of its 126 MB for their K and V; above it, sequence by sequence in ascending order: the last
// query chunk first cost 8 x 256 chunks 1711 -> 1749 us forward + backward, the forward at 1 x 1,024 chunks, K = 16 364 -> 377.
template <class Args>
inline bool late_chunks_first(const Args& a) {
  return (long long)a.N * a.C * a.Hkv * a.L * a.D * 2 * 2 <= (64ll << 20);
}

// Warps of a kernel with that many registers a thread (a multiple of eight) that an SM holds: each of its four quarters has registers of its own.
constexpr int warps_per_sm(int regs) { return 4 * (512 / regs); }

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// The entry points run on the device that HOLDS THE BUFFERS, whatever the calling thread's
// current device is (PyTorch calls the backward from an autograd worker thread; a plain C caller
// may never have called cudaSetDevice).  DeviceScope finds the device of a device pointer,
// makes it current for the duration of the call and restores the previous one.
struct DeviceScope {
  int prev = -1, dev = -1, rc = 0;
  explicit DeviceScope(const void* device_ptr);
  ~DeviceScope();
  DeviceScope(const DeviceScope&) = delete;
  DeviceScope& operator=(const DeviceScope&) = delete;
};
// Number of SMs of a device (asked once per device).
int sm_count(int dev);

// Argument rules shared by lmk_score_topk, lmk_topk_workspace_bytes and lmk_score_topk_static.
int check_topk(const LmkTopkArgs* a);

}  // namespace gca
