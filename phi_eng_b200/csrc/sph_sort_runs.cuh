// Placement of the general bucket sort, shared by the 2D and 3D kernel chains
// (the scan before it: sph_kernels.cu). start[k] = first slot of bucket k; count
// holds the buckets' sizes and is zero again afterwards.
//
// The gather functor writes a particle's sorted entries: ga(slot, key, id), which
// is ga.load(id) and ga.store(slot, key, id, row).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sph_chain.cuh"
#include "sph_kernels.h"
#include "sph_warp.cuh"

namespace phieng {

// Longest bucket k_place_runs finishes by itself (a word of run marks).
constexpr uint32_t kRunMax = 32;

// One particle per thread in the previous sort's slot order (prev[s] = id).
// Particles keep their cell from one substep to the next almost always, so most
// buckets arrive as one run of consecutive slots: where the run of equal keys
// around a slot is as long as its bucket, the particle's rank is the number of
// smaller tags in the run, and it is gathered into its final slot at once. Every
// thread of the run comes to the same conclusion from the same slots, so this
// takes no atomics. The particles of the other buckets take any slot of their
// bucket (tkey, tid) and are listed for k_fix_list. With order tags the sentinel
// bucket is always left to k_fix_list: unused rows of a rank world share one tag.
//
// Against a slot by an atomic for every particle and a ranking kernel over all of
// them: 2^20 particles 14.1 -> 12.4 + 2.1 us (the second kernel's launch), 512
// scenes of 9,040 132 -> 58.6 + 2.3 us, 100^3 particles in 3D 26 -> 20.2 + 2.3 us.
// Issue-bound when each thread walked its run in shared memory (261 instructions
// a warp, 14.0 us at 2^20), so the runs' borders are marked in one word a warp (head: the
// slot before holds another key) and found by bit scans, and the tags are only
// compared where a second word says that they do not rise along the run: a run
// that nobody entered is still in its last sort's order.
template <class Gather>
__global__ void __launch_bounds__(256) k_place_runs(const uint32_t* __restrict__ key,
                                                    const uint32_t* __restrict__ prev, uint32_t n,
                                                    uint32_t* __restrict__ count, const uint32_t* __restrict__ start,
                                                    const uint32_t* __restrict__ order, uint32_t* __restrict__ tkey,
                                                    uint32_t* __restrict__ tid_out, uint32_t* __restrict__ list,
                                                    uint32_t* __restrict__ list_n, uint32_t sentinel, Gather ga) {
  static_assert(kRunMax == 32u, "a halo warp on either side of the block's slots, one word of marks each");
  constexpr uint32_t kSpan = 256u + 2u * kRunMax, kWords = kSpan / 32u;
  __shared__ uint32_t s_key[kSpan], s_tag[kSpan];
  __shared__ uint32_t s_head[kWords], s_fall[kWords];
  __shared__ uint32_t s_open, s_base;
  chain_wait(key, prev, start, order);
  const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
  const uint32_t s = blockIdx.x * 256u + t, i = t + kRunMax;
  if (t == 0) s_open = 0u;
  // the particle's row and its bucket's range are on their way while the block
  // waits for its keys: they depend on the id alone
  uint32_t id = 0u, k = 0xFFFFFFFFu, tag = 0u, lo = 0u, hi = 0u;
  typename Gather::Row row{};
  if (s < n) {
    id = prev[s];
    k = key[id];
    row = ga.load(id);
    tag = order ? order[id] : id;
    lo = start[k];
    hi = start[k + 1];
  }
  s_key[i] = k;
  s_tag[i] = tag;
  const uint32_t ih = w == 0 ? lane : 256u + t;  // warps 0 and 1: also a halo slot
  if (w < 2) {
    const uint32_t sh = blockIdx.x * 256u + ih - kRunMax;  // wraps below 0: not < n
    uint32_t kh = 0xFFFFFFFFu, th = 0u;
    if (sh < n) {
      th = prev[sh];
      kh = key[th];
      if (order) th = order[th];
    }
    s_key[ih] = kh;
    s_tag[ih] = th;
  }
  __syncthreads();
  {
    const bool head = s_key[i - 1u] != k;
    const uint32_t h = __ballot_sync(0xFFFFFFFFu, head);
    const uint32_t f = __ballot_sync(0xFFFFFFFFu, !head && s_tag[i - 1u] >= tag);
    if (lane == 0) {
      s_head[w + 1u] = h;
      s_fall[w + 1u] = f;
    }
  }
  if (w < 2) {
    // the first halo slot counts as a head: a run from before it that reaches
    // the block's slots is longer than kRunMax
    const bool head = ih == 0u || s_key[ih - 1u] != s_key[ih];
    const uint32_t h = __ballot_sync(0xFFFFFFFFu, head);
    const uint32_t f = __ballot_sync(0xFFFFFFFFu, !head && s_tag[ih - 1u] >= s_tag[ih]);
    if (lane == 0) {
      s_head[w == 0 ? 0u : kWords - 1u] = h;
      s_fall[w == 0 ? 0u : kWords - 1u] = f;
    }
  }
  __syncthreads();
  bool open = false;
  if (s < n) {
    // marks of the 32 slots up to this one (its own in bit 31) and of the next 32
    const uint32_t h1 = s_head[w + 1u], f1 = s_fall[w + 1u];
    const uint32_t hb = __funnelshift_rc(s_head[w], h1, lane + 1u), ha = __funnelshift_rc(h1, s_head[w + 2u], lane + 1u);
    const uint32_t d = (uint32_t)__clz((int)hb);              // slots of the run before this one
    const uint32_t e = (uint32_t)__ffs((int)ha) - 1u;         // slots of the run after this one
    open = hb == 0u || ha == 0u || d + e + 1u != hi - lo || hi - lo > kRunMax || (order && k == sentinel);
    if (!open) {
      const uint32_t fb = __funnelshift_rc(s_fall[w], f1, lane + 1u);
      const uint32_t fa = __funnelshift_rc(f1, s_fall[w + 2u], lane + 1u);
      uint32_t rank = d;
      if ((fb >> (31u - d)) | (fa & ((1u << e) - 1u))) {
        rank = 0u;
        for (uint32_t q = i - d; q <= i + e; q++) rank += s_tag[q] < tag ? 1u : 0u;
      }
      if (d == 0u) count[k] = 0u;
      ga.store(lo + rank, k, id, row);
    }
  }
  // the others: a few by an atomic each, many (dense buckets, the sentinel's) by
  // one per run of equal keys; one per warp for the block's part of the list
  const uint32_t act = __ballot_sync(0xFFFFFFFFu, open);
  uint32_t mine = 0u, slot = 0u;
  if (open) {
    if (__popc(act) <= 8) {
      slot = lo + atomicSub(&count[k], 1u) - 1u;
    } else {
      uint32_t first, len, rank;
      key_run(act, k, lane, &first, &len, &rank);
      uint32_t left = 0u;
      if (first == lane) left = atomicSub(&count[k], len);
      slot = lo + __shfl_sync(act, left, first) - len + rank;
    }
    tkey[slot] = k;
    tid_out[slot] = id;
    const uint32_t leader = (uint32_t)__ffs((int)act) - 1u;
    if (lane == leader) mine = atomicAdd(&s_open, (uint32_t)__popc(act));
    mine = __shfl_sync(act, mine, leader) + (uint32_t)__popc(act & ((1u << lane) - 1u));
  }
  __syncthreads();
  if (t == 0 && s_open) s_base = atomicAdd(list_n, s_open);
  __syncthreads();
  if (open) list[s_base + mine] = slot;
}

// One particle per thread in id order, into any slot of its bucket.
static __global__ void __launch_bounds__(256) k_place_all(const uint32_t* __restrict__ key, uint32_t n,
                                                   uint32_t* __restrict__ count, const uint32_t* __restrict__ start,
                                                   uint32_t* __restrict__ tkey, uint32_t* __restrict__ tid_out) {
  chain_wait(key, start);
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= n) return;
  const uint32_t k = key[id];
  // one atomic per run of equal keys in consecutive lanes
  const uint32_t act = __activemask();
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t first, len, rank;
  key_run(act, k, lane, &first, &len, &rank);
  uint32_t left = 0;
  if (first == lane) left = atomicSub(&count[k], len);
  left = __shfl_sync(act, left, first);
  const uint32_t slot = start[k] + left - len + rank;
  tkey[slot] = k;
  tid_out[slot] = id;
}

// Final slot = bucket start + rank of the id (or its order tag) among the
// bucket's, for the particle placed in slot s. With order tags, the sentinel
// bucket of non-finite particles keeps its placement slots: no walk visits it,
// and its size (a rank world's unused slots) would make ranking quadratic.
template <class Gather>
__device__ __forceinline__ void fix_slot(uint32_t s, const uint32_t* __restrict__ tkey,
                                         const uint32_t* __restrict__ tid_in, const uint32_t* __restrict__ start,
                                         const uint32_t* __restrict__ order, uint32_t sentinel, const Gather& ga) {
  const uint32_t k = tkey[s], id = tid_in[s];
  if (order && k == sentinel) {
    ga(s, k, id);
    return;
  }
  const uint32_t lo = start[k], hi = start[k + 1];
  uint32_t rank = 0;
  if (order) {
    const uint32_t tag = order[id];
    for (uint32_t j = lo; j < hi; j++) rank += order[tid_in[j]] < tag ? 1u : 0u;
  } else {
    for (uint32_t j = lo; j < hi; j++) rank += tid_in[j] < id ? 1u : 0u;
  }
  ga(lo + rank, k, id);
}

template <class Gather>
__global__ void __launch_bounds__(256) k_fix_list(const uint32_t* __restrict__ list,
                                                  const uint32_t* __restrict__ list_n,
                                                  const uint32_t* __restrict__ tkey,
                                                  const uint32_t* __restrict__ tid_in,
                                                  const uint32_t* __restrict__ start,
                                                  const uint32_t* __restrict__ order, uint32_t sentinel, Gather ga) {
  chain_wait(list, list_n, tkey, tid_in, start, order);
  const uint32_t m = *list_n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    fix_slot(list[i], tkey, tid_in, start, order, sentinel, ga);
}

template <class Gather>
__global__ void __launch_bounds__(256) k_fix_all(uint32_t n, const uint32_t* __restrict__ tkey,
                                                 const uint32_t* __restrict__ tid_in,
                                                 const uint32_t* __restrict__ start,
                                                 const uint32_t* __restrict__ order, uint32_t sentinel, Gather ga) {
  chain_wait(tkey, tid_in, start, order);
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) fix_slot(s, tkey, tid_in, start, order, sentinel, ga);
}

// Sort of n particles with keys in [0, m) by (key, id or tag); the scan resets
// the list's length.
template <class Gather>
inline void enqueue_bucket_sort(const BucketSort& bs, uint32_t n, uint32_t m, bool by_slot, const Gather& ga,
                                cudaStream_t st) {
  const uint32_t blocks = (n + 255u) / 256u;
  enqueue_bucket_scan(bs, m, st);
  if (by_slot) {
    launch_chained(k_place_runs<Gather>, blocks, 256, 0, st, bs.key, bs.prev, n, bs.count, bs.start, bs.order, bs.tkey,
                   bs.tid, bs.list, bs.list_n, m - 1u, ga);
    launch_chained(k_fix_list<Gather>, blocks < 592u ? blocks : 592u, 256, 0, st, bs.list, bs.list_n, bs.tkey, bs.tid,
                   bs.start, bs.order, m - 1u, ga);
  } else {
    launch_chained(k_place_all, blocks, 256, 0, st, bs.key, n, bs.count, bs.start, bs.tkey, bs.tid);
    launch_chained(k_fix_all<Gather>, blocks, 256, 0, st, n, bs.tkey, bs.tid, bs.start, bs.order, m - 1u, ga);
  }
}

}  // namespace phieng
