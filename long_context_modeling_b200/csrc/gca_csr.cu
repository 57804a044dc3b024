// Inverse retrieval index for the kv-major backward pass.
//
// For every cache chunk (n, c) the backward needs the list of (query chunk j, slot k)
// pairs that retrieved it, in a fixed order so that float32 accumulation is reproducible.
// Each valid entry becomes the 64-bit key  (n*C + c) << 32 | (j*K + k); a stable radix sort
// on the chunk field gives the lists back to back (two 8-bit passes at N*C = 2048 instead of
// the eight of a full 64-bit sort), and a binary search per chunk finds where each list starts.
// Padding slots (index < 0) and out-of-range indices sort to the end.  Problems of a training step's size take a
// single launch with the same result (csr_list_kernel).
#include <cstdlib>

#include <cub/device/device_radix_sort.cuh>

#include "gca_common.cuh"

namespace gca {

namespace {

__global__ void csr_keys_kernel(const int32_t* __restrict__ indices, unsigned long long* __restrict__ keys,
                                int N, int JK, int C) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)N * JK) return;
  const int n = (int)(i / JK);
  const int t = (int)(i % JK);
  const int idx = indices[i];
  keys[i] = (idx < 0 || idx >= C) ? ~0ull
                                  : (((unsigned long long)((long long)n * C + idx)) << 32) | (unsigned)t;
}

__device__ __forceinline__ long long csr_lower_bound(const unsigned long long* __restrict__ sorted, long long total,
                                                     unsigned long long target) {
  long long lo = 0, hi = total;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (sorted[mid] < target) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// A thread emits a chunk's entry of the kv-major walking order: key = sequence (by_count: 0) << cbits | (cmax - count), so that an
// ascending sort lists a sequence's (all) chunks by decreasing number of retrievers; value =
// (first entry, one past the last, chunk id): what the kv-major kernel reads per unit.
__global__ void csr_units_kernel(const unsigned long long* __restrict__ sorted, int* __restrict__ tickets, unsigned* __restrict__ ukeys,
                                 int4* __restrict__ uvals, long long total, long long NC, int C, int cbits, unsigned cmax, bool by_count) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < 2) tickets[c] = 0;
  if (c >= NC) return;
  const long long lo = csr_lower_bound(sorted, total, (unsigned long long)c << 32);
  const unsigned cnt = (unsigned)(csr_lower_bound(sorted, total, (unsigned long long)(c + 1) << 32) - lo);
  ukeys[c] = (by_count ? 0u : (unsigned)(c / C) << cbits) | (cmax - (cnt < cmax ? cnt : cmax));
  uvals[c] = make_int4((int)lo, (int)lo + (int)cnt, (int)c, 0);
}

// ---------------------------------------------------------------------------------------------
// Problems of a training step's size: the whole index in ONE launch of small blocks, bit-identical to the radix-sort path
// below, which costs nine launches (~85 us).  A block handles eight chunks of a sequence; its warps read a section of the
// sequence's J*K entries each, twice:
//   1. counting the retrievers of ALL the sequence's chunks (shared-memory histogram; redundant between blocks, but J*K
//      reads from L2 are nothing) and of the block's own chunks per section.  That gives every list its start -- lists of
//      a sequence lie back to back from entry n * J * K --, its place in the walking order (chunks by decreasing count,
//      ties by id), and every section its first entry of every list;
//   2. writing the entries that name one of the block's chunks, in order.
// What bounds it is the chain of loads: 16 are in flight per lane.  Few registers, 4 bytes of shared memory per chunk: its
// blocks run BESIDE the q-major pass, which is launched while they work (nothing in it depends on the index) and fills
// the SMs to all but this.  In front of the q-major pass (one block per sequence, 145 KB of shared memory) it took 14 us
// at 8 x 256 chunks, K = 8, and 34 us at 1,024 chunks, K = 16.
constexpr int LIST_WARPS = 8, LIST_MAX_C = 2048, LIST_LOADS = 16;

__global__ void __launch_bounds__(LIST_WARPS * 32)
csr_list_kernel(const int32_t* __restrict__ indices, unsigned long long* __restrict__ keys_out, int4* __restrict__ unit_tab, int* __restrict__ tickets,
                int JK, int C, bool by_count) {
  __shared__ int cnt[LIST_MAX_C];
  __shared__ int sect[LIST_WARPS][LIST_WARPS];       // [section][chunk of this block]: entries, then the first one's place
  const int n = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int32_t* row = indices + (long long)n * JK;
  for (int i = threadIdx.x; i < C; i += LIST_WARPS * 32) cnt[i] = 0;
  if (threadIdx.x < LIST_WARPS * LIST_WARPS) (&sect[0][0])[threadIdx.x] = 0;
  pdl_wait();
  pdl_trigger();                         // everything before this kernel is complete: the next one may start
  if (blockIdx.x == 0 && n == 0 && threadIdx.x < 2) tickets[threadIdx.x] = 0;
  __syncthreads();
  const int c0 = blockIdx.x * LIST_WARPS, c1 = min(c0 + LIST_WARPS, C);
  const int per = ((JK + LIST_WARPS * 32 - 1) / (LIST_WARPS * 32)) * 32, first = warp * per, last = min(first + per, JK);
  for (int t0 = first; t0 < last; t0 += 32 * LIST_LOADS) {
    int v[LIST_LOADS];
#pragma unroll
    for (int x = 0; x < LIST_LOADS; ++x) v[x] = t0 + 32 * x + lane < last ? row[t0 + 32 * x + lane] : -1;
#pragma unroll
    for (int x = 0; x < LIST_LOADS; ++x) {
      if (v[x] >= 0 && v[x] < C) atomicAdd(&cnt[v[x]], 1);
      if (v[x] >= c0 && v[x] < c1) atomicAdd(&sect[warp][v[x] - c0], 1);
    }
  }
  __syncthreads();
  const int c = c0 + warp;
  if (c < c1) {
    const int mine = cnt[c];
    int start = 0, rank = 0;
    for (int i = lane; i < C; i += 32) {
      const int v = cnt[i];
      start += i < c ? v : 0;
      rank += v > mine || (v == mine && i < c);
    }
#pragma unroll
    for (int of = 16; of > 0; of >>= 1) {
      start += __shfl_xor_sync(0xffffffffu, start, of);
      rank += __shfl_xor_sync(0xffffffffu, rank, of);
    }
    start += n * JK;
    if (lane == 0) {
      unit_tab[by_count ? (long long)rank * gridDim.y + n : (long long)n * C + rank] = make_int4(start, start + mine, n * C + c, 0);
      for (int w = 0; w < LIST_WARPS; ++w) {
        const int here = sect[w][warp];
        sect[w][warp] = start;
        start += here;
      }
    }
  }
  __syncthreads();
  for (int t0 = first; t0 < last; t0 += 32 * LIST_LOADS) {
    int v[LIST_LOADS];
#pragma unroll
    for (int x = 0; x < LIST_LOADS; ++x) v[x] = t0 + 32 * x + lane < last ? row[t0 + 32 * x + lane] : -1;
#pragma unroll
    for (int x = 0; x < LIST_LOADS; ++x) {
      const bool hit = v[x] >= c0 && v[x] < c1;
      if (!__any_sync(0xffffffffu, hit)) continue;
      const unsigned same = __match_any_sync(0xffffffffu, hit ? v[x] : -1), before = same & ((1u << lane) - 1u);
      const int at = hit ? sect[warp][v[x] - c0] : 0;
      if (hit) keys_out[at + __popc(before)] = (unsigned long long)((long long)n * C + v[x]) << 32 | (unsigned)(t0 + 32 * x + lane);
      __syncwarp();
      if (hit && before == 0) sect[warp][v[x] - c0] = at + __popc(same);
      __syncwarp();
    }
  }
}

// Beyond 2^27 (blocks x entries x 8, a few tens of microseconds of L2 reads) or 2,048 chunks per sequence: the sort.
bool small_path(int N, int JK, int C) {
  return C <= LIST_MAX_C && (long long)N * JK < (1ll << 31) && (long long)N * C * JK <= (1ll << 27) && N <= 65535;
}

// For passes that do not write it themselves.  (The bf16 tensor-core passes of one call do: 109 row blocks x 8 heads, forward + backward, calls in
// a row 79.5 -> 76.3 us.)
__global__ void csr_identity_kernel(Csr index, int NC, int C) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 2) index.tickets[i] = 0;
  if (i < NC) identity_entry(index, i, C);
}

size_t cub_temp_bytes(long long total) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortKeys(nullptr, bytes, (const unsigned long long*)nullptr,
                                 (unsigned long long*)nullptr, (int)total);
  return bytes;
}

size_t cub_pairs_temp_bytes(long long n) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned*)nullptr, (unsigned*)nullptr,
                                  (const int4*)nullptr, (int4*)nullptr, (int)n);
  return bytes;
}

int bits_for(long long v) {       // smallest b with 2^b > v
  int b = 0;
  while ((1ll << b) <= v) ++b;
  return b;
}

}  // namespace

size_t csr_workspace_bytes(int N, int J, int K, int C) {
  const long long total = (long long)N * J * K;
  const long long NC = (long long)N * C;
  return align_up(total * 8, 256) * 2 + align_up(cub_temp_bytes(total), 256) +
         align_up(NC * 4, 256) * 2 + align_up(NC * 16, 256) * 2 + align_up(cub_pairs_temp_bytes(NC), 256) + 256;
}

int build_csr(const int32_t* indices, int N, int J, int K, int C, void* workspace, size_t workspace_bytes,
              bool by_count, Csr* out, size_t* used_bytes, cudaStream_t stream, bool launch, bool by_sort) {
  const long long total = (long long)N * J * K;
  const long long NC = (long long)N * C;
  if (total >= (1ll << 31) || NC >= (1ll << 31)) return GCA_ERR_TOO_LARGE;
  const size_t need = csr_workspace_bytes(N, J, K, C);
  if (!workspace || workspace_bytes < need) return GCA_ERR_WORKSPACE;
  char* p = (char*)workspace;
  unsigned long long* keys_in = (unsigned long long*)p;  p += align_up(total * 8, 256);
  unsigned long long* keys_out = (unsigned long long*)p; p += align_up(total * 8, 256);
  size_t temp = cub_temp_bytes(total);
  void* temp_ptr = p;                                    p += align_up(temp, 256);
  unsigned* ukeys_in = (unsigned*)p;                     p += align_up(NC * 4, 256);
  unsigned* ukeys_out = (unsigned*)p;                    p += align_up(NC * 4, 256);
  int4* uvals_in = (int4*)p;                             p += align_up(NC * 16, 256);
  int4* uvals_out = (int4*)p;                            p += align_up(NC * 16, 256);
  size_t utemp = cub_pairs_temp_bytes(NC);
  void* utemp_ptr = p;                                   p += align_up(utemp, 256);
  int* tickets = (int*)p;
  // a chunk has at most J*K retrievers; the unit key holds (J*K - count) below the sequence number
  const long long cmax = (long long)J * K;
  const int cbits = bits_for(cmax), nbits = bits_for(N);
  if (cbits + nbits > 32) return GCA_ERR_TOO_LARGE;
  out->overlaps = false;
  if (launch && !indices && NC > 0) {
    GCA_CUDA_CHECK(launch_dependent(csr_identity_kernel, dim3((unsigned)((NC + 255) / 256)), dim3(256), 0, stream, Csr{keys_out, uvals_out, tickets, false}, (int)NC, C));
    out->overlaps = true;
  } else if (launch && NC > 0 && total > 0 && !by_sort && small_path(N, J * K, C)) {
    GCA_CUDA_CHECK(launch_dependent(csr_list_kernel, dim3((unsigned)((C + LIST_WARPS - 1) / LIST_WARPS), (unsigned)N), dim3(LIST_WARPS * 32), 0,
                                    stream, indices, keys_out, uvals_out, tickets, J * K, C, by_count));
    out->overlaps = true;
  } else if (launch) {
    if (total > 0) {
      csr_keys_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(indices, keys_in, N, J * K, C);
      GCA_CUDA_CHECK(cudaGetLastError());
      // The keys are generated in increasing (j*K + k) order inside a sequence, and the radix sort
      // is stable, so sorting on the chunk field alone is a full sort.  Valid chunk ids are < N*C
      // <= 2^b; the all-ones key of an invalid entry has bit b set and sorts behind them.
      int b = 0;
      while ((1ll << b) < NC) ++b;
      const int end_bit = 32 + b + 1 > 64 ? 64 : 32 + b + 1;
      GCA_CUDA_CHECK(cub::DeviceRadixSort::SortKeys(temp_ptr, temp, keys_in, keys_out, (int)total, 32, end_bit, stream));
    }
    if (NC > 0) {
      csr_units_kernel<<<(unsigned)((NC + 255) / 256), 256, 0, stream>>>(keys_out, tickets, ukeys_in, uvals_in, total, NC, C, cbits,
                                                                         (unsigned)cmax, by_count);
      GCA_CUDA_CHECK(cudaGetLastError());
      GCA_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(utemp_ptr, utemp, ukeys_in, ukeys_out, uvals_in, uvals_out, (int)NC, 0,
                                                     cbits + nbits, stream));
    }
  }
  out->sorted_keys = keys_out;
  out->unit_tab = uvals_out;
  out->tickets = tickets;
  *used_bytes = need;
  return 0;
}

}  // namespace gca
