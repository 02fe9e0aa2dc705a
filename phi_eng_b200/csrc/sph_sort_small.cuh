// Bucket sort of a small particle set in one launch, shared by the 2D and 3D
// kernel chains.
//
// The general sort (sph_kernels.cu) is four dependent launches, each near the
// few microseconds a launch costs whatever its size: on a 4,096-particle world
// scan 6.4, place 4.6 and rank 3.1 us. Here every block sorts the whole set by
// bucket in its own shared memory: histogram of the keys (the atomic's return
// value is the particle's arrival rank in its bucket), exclusive scan, ids to
// their bucket's slots. Each block then ranks by id and gathers the buckets that
// start in its share of the slots (an arrival order is its own block's, a
// bucket's particles are the same for all), writes its share of the range table
// and clears its share of the counts. The result is the general sort's: order
// (key, id), start[b] = first slot of bucket b for b in [0, m], and the bucket
// counts cleared for the force pass.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "sph_chain.cuh"

namespace phieng {

constexpr uint32_t kSmallSortMax = 8192;      // particles: eight per thread
constexpr uint32_t kSmallSortKeys = 17 * 1024;  // keys (buckets and the sentinel)

inline bool small_sort_applies(uint32_t n, uint32_t m) { return n <= kSmallSortMax && m <= kSmallSortKeys; }

inline size_t small_sort_smem(uint32_t n, uint32_t m) {
  return sizeof(uint32_t) * ((size_t)(m + 1023) / 1024 * 1024 + 2 * (((size_t)n + 31) / 32 * 32));
}

// Word of entry k in a shared array: the low five bits are mixed with higher
// ones, since consecutive particles often differ by a power of two of buckets
// or slots (a lattice stored z first), which would put a warp on one bank.
__device__ __forceinline__ uint32_t small_sort_word(uint32_t k) { return k ^ (((k >> 5) ^ (k >> 10)) & 31u); }

// ga(slot, key, id) writes the sorted entries of a particle. count (if not
// null) is cleared: count_len entries, a multiple of four.
template <class Gather>
__global__ void __launch_bounds__(1024) k_sort_small(const uint32_t* __restrict__ key, uint32_t n, uint32_t m,
                                                     uint32_t* __restrict__ start, uint32_t* __restrict__ count,
                                                     uint32_t count_len, Gather ga) {
  chain_wait(key);
  extern __shared__ uint32_t sort_small_smem[];
  __shared__ uint32_t warp_tot[32];
  constexpr int kPer = kSmallSortMax / 1024;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  const uint32_t chunk = (m + 1023u) / 1024u;  // keys per thread in the scan
  uint32_t* cur = sort_small_smem;
  uint32_t* ids = cur + chunk * 1024u;  // by bucket, then arrival
  uint32_t* keys = ids + (n + 31u) / 32u * 32u;
  const uint32_t gtid = blockIdx.x * 1024u + tid, gstep = gridDim.x * 1024u;
  uint32_t k[kPer], a[kPer];
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const uint32_t i = tid + q * 1024u;
    if (i < n) k[q] = key[i];
  }
  for (uint32_t i = tid; i < chunk * 1024u; i += 1024u) cur[i] = 0u;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; q++)
    if (tid + q * 1024u < n) a[q] = atomicAdd(&cur[small_sort_word(k[q])], 1u);
  __syncthreads();
  uint32_t sum = 0;
  for (uint32_t q = 0; q < chunk; q++) sum += cur[small_sort_word(tid * chunk + q)];
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint32_t t = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, t, o);
      if (lane >= (uint32_t)o) t += y;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  uint32_t run = x - sum + (wid ? warp_tot[wid - 1] : 0u);
  for (uint32_t q = 0; q < chunk; q++) {
    uint32_t& word = cur[small_sort_word(tid * chunk + q)];
    const uint32_t c = word;
    word = run;
    run += c;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const uint32_t i = tid + q * 1024u;
    if (i < n) {
      const uint32_t at = small_sort_word(cur[small_sort_word(k[q])] + a[q]);
      ids[at] = i;
      keys[at] = k[q];
    }
  }
  for (uint32_t i = gtid; i <= m; i += gstep) start[i] = i < m ? cur[small_sort_word(i)] : n;
  if (count)
    for (uint32_t i = gtid; 4u * i < count_len; i += gstep)
      reinterpret_cast<uint4*>(count)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const uint32_t share = (n + gridDim.x - 1u) / gridDim.x, first = blockIdx.x * share, end = first + share;
  for (uint32_t f = first + tid; f < n; f += 1024u) {
    const uint32_t kf = keys[small_sort_word(f)];
    const uint32_t lo = cur[small_sort_word(kf)];
    if (lo >= end) break;     // this bucket and the later ones are other blocks'
    if (lo < first) continue;  // as is one that began before this share
    const uint32_t hi = kf + 1u < m ? cur[small_sort_word(kf + 1u)] : n;
    const uint32_t id = ids[small_sort_word(f)];
    uint32_t rank = 0;
    for (uint32_t j = lo; j < hi; j++) rank += ids[small_sort_word(j)] < id ? 1u : 0u;
    ga(lo + rank, kf, id);
  }
}

template <class Gather>
inline void launch_sort_small(const uint32_t* key, uint32_t n, uint32_t m, uint32_t* start, uint32_t* count,
                              uint32_t count_len, const Gather& ga, cudaStream_t st) {
  const size_t smem = small_sort_smem(n, m);
  // the limit is the kernel's, shared by all threads and worlds: always the
  // largest set's, never this set's need
  cudaFuncSetAttribute(k_sort_small<Gather>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)small_sort_smem(kSmallSortMax, kSmallSortKeys));
  launch_chained(k_sort_small<Gather>, std::max<uint32_t>(1u, (n + 1023u) / 1024u * 4u), 1024, smem, st, key, n, m,
                 start, count, count_len, ga);
}

}  // namespace phieng
