// Whole 2D steps of a small world in one launch, included by sph_kernels.cu
// inside its anonymous namespace.
//
// The chain of five launches takes ~25 us per substep on a 4,096-particle world
// and no less on 96 particles: every launch waits for the one before it and
// leaves most of the 148 SMs idle. Here one thread-block cluster takes the
// world through any number of steps. Each block owns an equal share of the
// sorted slots. Per substep it
//   - sorts: bucket histogram of all keys and its scan in shared memory (every
//     block for itself), then the particles of the bucket rows that its share's
//     neighbours can lie in (its window) into (key, id) order;
//   - computes its share's density, one thread per particle, and lists each
//     particle's neighbours in visit order;
//   - meets the others at the cluster's barrier and reads its window's densities
//     from their shared memory;
//   - computes force and integrates with kSmallLanes lanes per particle, which
//     evaluate its pairs side by side and sum the terms over shared memory in
//     the visit order; writes the new states and keys to global memory; meets
//     the others again.
// Every sum keeps its order, so every result has the bits of the one-thread
// passes, in both arithmetic modes.
//
// Per substep 8.7 us for 64 particles, 13.5 for 4,096 (25 with the launches). What
// is left is the instructions of one particle's chain (density ~4,000 cycles,
// pairs 3,200 to 5,300, integrate 3,000 for a particle in contact with two
// walls) and, above 2,000 particles, their issue on 16 SMs.
//
// A step's CFL substep count (cfl_substeps, fluid.rs:562-588) is computed here
// with the host's f32 arithmetic, so such a world needs no host read per step.
constexpr uint32_t kSmallMax = 4096;       // particles
constexpr uint32_t kSmallKeys = 9 * 1024;  // bucket keys
constexpr uint32_t kSmallLanes = 4;
constexpr uint32_t kSmallBlocks = 16;  // blocks of the largest cluster
constexpr uint32_t kSmallShare = kSmallMax / kSmallBlocks;  // slots of a block at most
constexpr uint32_t kSmallList = 32;    // listed neighbours of a particle (11.6 at rest density)
constexpr uint32_t kSmallBodies = 32;  // static bodies (kept in shared memory)
constexpr int kSmallPer = 4;           // particles per thread of the sort

struct SmallCfl {
  uint32_t on;  // 0: one substep per step
  uint32_t max_substeps;
  float c0, cfl_h;  // sound speed, cfl * max(h, EPS)
};

struct SmallArgs {
  float4* state;
  const float* mass;      // id order (F_MASS)
  const uint8_t* phase;   // id order (F_PHASE)
  const DevBody* bodies;
  // left as the chain of launches leaves them after the last substep
  uint32_t* sid;
  float2* sdq;
  float* spres;
  uint32_t* key;
  uint32_t* count;
  uint32_t count_len;
  unsigned long long* substeps;       // += substeps taken (null: not counted)
  unsigned long long* substeps_host;  // the new total, in page-locked host memory
  uint32_t n, steps;
  float dt;  // of a step (before CFL substeps)
  SmallCfl cfl;
};

// Blocks of the cluster and threads of a block: 64 slots a block until there
// are 16 (exact step of 256 / 1,023 particles: 9.2 / 10.4 us, with 256 slots a
// block 11.9 / 12.3), then up to 256, with kSmallLanes threads a slot; so at
// most kSmallPer particles per thread.
struct SmallShape {
  uint32_t blocks, share, threads;
};
inline SmallShape small_shape(uint32_t n) {
  SmallShape s;
  s.blocks = 1;
  while (s.blocks < kSmallBlocks && s.blocks * 64u < n) s.blocks *= 2;
  s.share = (n + s.blocks - 1u) / s.blocks;
  s.threads = std::max(256u, (s.share * kSmallLanes + 31u) / 32u * 32u);
  return s;
}

// Word offsets of the shared arrays, each 16-byte aligned. work: the window's
// particles by arrival, then the pair terms; nl: neighbour lists,
// [kSmallList + 1][share] (the last row takes what does not fit); cnt: their
// lengths.
struct SmallLayout {
  uint32_t work, cur, sid, skey, spos, svel, sdq, smass, sphase, nl, cnt, words;
};

__host__ __device__ inline SmallLayout small_layout(uint32_t n, uint32_t m, uint32_t share, uint32_t threads,
                                                    bool mass, bool phase, bool plain) {
  const uint32_t np = (n + 31u) / 32u * 32u;
  SmallLayout L;
  uint32_t at = 0;
  auto take = [&](uint32_t words) {
    const uint32_t r = at;
    at += (words + 3u) / 4u * 4u;
    return r;
  };
  const uint32_t tw = threads * (plain ? 6u : 8u);
  L.work = take(tw > np ? tw : np);
  // the scan deals (m + threads - 1) / threads keys to a thread; the swizzle
  // moves a word inside its 32
  L.cur = take(((m + threads - 1u) / threads * threads + 31u) / 32u * 32u);
  L.sid = take((share + 1u) / 2u);
  L.skey = take((share + 1u) / 2u);
  L.spos = take(2u * np);
  L.svel = take(2u * np);
  L.sdq = take(2u * np);
  L.smass = take(mass ? np : 0u);
  L.sphase = take(phase ? (share + 3u) / 4u : 0u);
  L.nl = take(((kSmallList + 1u) * share + 1u) / 2u);
  L.cnt = take(share);
  L.words = at;
  return L;
}

// Bytes of the largest world's shared arrays.
inline size_t small_smem_max() {
  return sizeof(uint32_t) *
         small_layout(kSmallMax, kSmallKeys, kSmallShare, kSmallShare * kSmallLanes, true, true, false).words;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// All threads of all blocks of the cluster; writes before it (global and
// shared, remote included) are visible after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float2 load_remote(const float2* local, uint32_t rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
  uint32_t r;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(r) : "memory");
  return v;
}

template <bool MASS, bool PHASE, bool PLAIN, bool FAST>
__global__ void __launch_bounds__(kSmallShare* kSmallLanes, 1)
    k_small_steps(SmallArgs A, const __grid_constant__ StepParams P) {
  extern __shared__ __align__(16) uint32_t small_smem[];
  __shared__ uint32_t warp_tot[32];
  __shared__ float s_max[32];
  __shared__ uint32_t s_key[2];  // buckets of the share's first and last slot
  __shared__ DevBody s_bodies[kSmallBodies];
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const uint32_t n = A.n, tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  const uint32_t threads = blockDim.x, warps = threads >> 5, per = (A.n + threads - 1u) / threads;
  const GridPlan& g = P.grid;
  const uint32_t m = g.sentinel + 1u, chunk = (m + threads - 1u) / threads;
  const uint32_t rank = cluster_rank(), blocks = cluster_size();
  const uint32_t share = (n + blocks - 1u) / blocks, first = min(rank * share, n), end = min(first + share, n);
  const SmallLayout L = small_layout(n, m, share, threads, MASS, PHASE, PLAIN);
  float* const terms = reinterpret_cast<float*>(small_smem + L.work);
  uint32_t* const cur = small_smem + L.cur;
  uint32_t* const ids = small_smem + L.work;
  uint16_t* const sid = reinterpret_cast<uint16_t*>(small_smem + L.sid);
  uint16_t* const skey = reinterpret_cast<uint16_t*>(small_smem + L.skey);
  float2* const spos = reinterpret_cast<float2*>(small_smem + L.spos);
  float2* const svel = reinterpret_cast<float2*>(small_smem + L.svel);
  float2* const sdq = reinterpret_cast<float2*>(small_smem + L.sdq);
  float* const smass = reinterpret_cast<float*>(small_smem + L.smass);
  uint8_t* const sphase = reinterpret_cast<uint8_t*>(small_smem + L.sphase);
  uint16_t* const nl = reinterpret_cast<uint16_t*>(small_smem + L.nl);
  uint32_t* const ncnt = small_smem + L.cnt;
  // the bodies: the barriers drop L1, where each read would cost an L2 round trip
  for (uint32_t i = tid; i < P.nbodies * (uint32_t)(sizeof(DevBody) / 4u); i += threads)
    reinterpret_cast<uint32_t*>(s_bodies)[i] = reinterpret_cast<const uint32_t*>(A.bodies + P.body_first)[i];
  // the bucket counts of the last substep's new keys accumulate from zero
  for (uint32_t i = rank * threads + tid; 4u * i < A.count_len; i += blocks * threads)
    reinterpret_cast<uint4*>(A.count)[i] = make_uint4(0u, 0u, 0u, 0u);
  cluster_sync();  // every block runs before any reads its shared memory
  auto start_of = [&](uint32_t k) { return k < m ? cur[small_sort_word(k)] : n; };
  uint32_t taken = 0;  // substeps so far
  for (uint32_t step = 0; step < A.steps; step++) {
    uint32_t ns = 1;
    float dt = A.dt;
    if (A.cfl.on) {
      // the step's substep count from the largest speed of all particles
      float v = 0.0f;
      for (uint32_t i = tid; i < n; i += threads) {
        const float4 q = __ldcg(&A.state[i]);
        const float l = __fsqrt_rn(__fadd_rn(__fmul_rn(q.z, q.z), __fmul_rn(q.w, q.w)));
        if (l > v) v = l;  // NaN never wins (f32::max)
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kAll, v, o));
      if (lane == 0) s_max[wid] = v;
      __syncthreads();
      v = lane < warps ? s_max[lane] : 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kAll, v, o));
      const float speed = __fadd_rn(A.cfl.c0, v);
      if (isfinite(speed) && speed > kEps) {
        const float dt_max = __fdiv_rn(A.cfl.cfl_h, speed);
        if (isfinite(dt_max) && dt_max > 0.0f) {
          const float c = ceilf(__fdiv_rn(A.dt, dt_max));
          ns = c >= (float)A.cfl.max_substeps ? A.cfl.max_substeps : c > 1.0f ? (uint32_t)c : 1u;
        }
      }
      dt = __fdiv_rn(A.dt, (float)ns);
    }
    for (uint32_t sub = 0; sub < ns; sub++) {
      const bool last = step + 1u == A.steps && sub + 1u == ns;
      // ---- keys (other blocks wrote them: past L1), histogram with arrival ranks
      uint32_t k[kSmallPer], a[kSmallPer];
#pragma unroll
      for (int u = 0; u < kSmallPer; u++) {
        const uint32_t i = tid + u * threads;
        if ((uint32_t)u < per && taken && i < n) k[u] = __ldcg(&A.key[i]);
      }
      if (taken == 0u) {
#pragma unroll 1
        for (int u = 0; u < (int)per; u++) {
          const uint32_t i = tid + u * threads;
          const float4 q = __ldcg(&A.state[min(i, n - 1u)]);
          const uint32_t kk = bucket_key(q.x, q.y, g);
#pragma unroll
          for (int t = 0; t < kSmallPer; t++)
            if (t == u) k[t] = kk;
        }
      }
      for (uint32_t i = tid; i < chunk * threads; i += threads) cur[small_sort_word(i)] = 0u;
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kSmallPer; u++)
        if ((uint32_t)u < per && tid + u * threads < n) a[u] = atomicAdd(&cur[small_sort_word(k[u])], 1u);
      __syncthreads();
      // ---- scan; the buckets that hold the share's first and last slot
      uint32_t sum = 0;
      for (uint32_t c = 0; c < chunk; c++) sum += cur[small_sort_word(tid * chunk + c)];
      uint32_t x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      if (lane == 31) warp_tot[wid] = x;
      __syncthreads();
      {
        uint32_t t = lane < wid ? warp_tot[lane] : 0u;
        t = __reduce_add_sync(kAll, t);
        uint32_t run = t + x - sum;
        for (uint32_t c = 0; c < chunk; c++) {
          uint32_t& word = cur[small_sort_word(tid * chunk + c)];
          const uint32_t v = word;
          word = run;
          if (first - run < v) s_key[0] = tid * chunk + c;  // run <= first < run + v
          if (end - 1u - run < v) s_key[1] = tid * chunk + c;
          run += v;
        }
      }
      __syncthreads();
      // ---- the window: the bucket rows one below the share's first to one
      // above its last; everything where those wrap (or the share is empty)
      uint32_t wlo = 0u, whi = n;
      if (first < end) {
        const uint32_t r0 = s_key[0] >> g.log2w, r1 = s_key[1] >> g.log2w;
        if (r0 >= 1u && r1 < g.maskh) {
          wlo = start_of((r0 - 1u) << g.log2w);
          whi = start_of((r1 + 2u) << g.log2w);
        }
      } else {
        whi = 0u;
      }
      uint32_t lo[kSmallPer], cnt[kSmallPer], most = 0;
      float4 q[kSmallPer];
#pragma unroll
      for (int u = 0; u < kSmallPer; u++) {
        cnt[u] = 0u;
        const uint32_t i = tid + u * threads;
        if ((uint32_t)u < per && i < n) {
          lo[u] = start_of(k[u]);
          if (lo[u] >= wlo && lo[u] < whi) {
            q[u] = __ldcg(&A.state[i]);
            cnt[u] = start_of(k[u] + 1u) - lo[u];
            most = max(most, cnt[u]);
            ids[small_sort_word(lo[u] + a[u])] = i;
            a[u] = 0u;  // from here the rank by id
          }
        }
      }
      __syncthreads();
      for (uint32_t t = 0; t < most; t++)
#pragma unroll
        for (int u = 0; u < kSmallPer; u++)
          if (t < cnt[u]) a[u] += ids[small_sort_word(lo[u] + t)] < tid + u * threads ? 1u : 0u;
#pragma unroll
      for (int u = 0; u < kSmallPer; u++)
        if (cnt[u]) {
          const uint32_t i = tid + u * threads, f = lo[u] + a[u];
          spos[f] = make_float2(q[u].x, q[u].y);
          svel[f] = make_float2(q[u].z, q[u].w);
          if (MASS) smass[f] = A.mass[i];
          if (f >= first && f < end) {
            sid[f - first] = (uint16_t)i;
            skey[f - first] = (uint16_t)k[u];
            if (PHASE) sphase[f - first] = A.phase[i];
          }
        }
      __syncthreads();
      // ---- density + EOS (k_density) and the neighbour lists, one thread per particle
      if (first + tid < end) {
        const uint32_t s = first + tid;
        const uint32_t ks = skey[tid];
        const float2 pi = spos[s];
        float rho = 0.0f;
        uint32_t c_nb = 0;
        if (ks != g.sentinel) {
          const uint32_t bx = ks & g.maskw, by = ks >> g.log2w;
          const bool seam = !(bx >= 1u && bx < g.maskw);
#pragma unroll 1
          for (uint32_t t = 0; t < (seam ? 9u : 3u); t++) {
            // row t, on the x seam bucket by bucket
            const uint32_t row = ((by + (seam ? t / 3u : t) - 1u) & g.maskh) << g.log2w;
            const uint32_t b0 = row + (seam ? ((bx + t % 3u - 1u) & g.maskw) : bx - 1u);
            const uint32_t rs = start_of(b0), re = start_of(b0 + (seam ? 1u : 3u));
#pragma unroll 1
            for (uint32_t j = rs; j < re; j += 4u) {  // four candidates in flight
              float2 c[4];
#pragma unroll
              for (uint32_t v = 0; v < 4; v++) c[v] = spos[min(j + v, re - 1u)];
#pragma unroll
              for (uint32_t v = 0; v < 4; v++) {
                const float dx = __fsub_rn(c[v].x, pi.x), dy = __fsub_rn(c[v].y, pi.y);
                const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
                const float w = neighbour_density_term<false>(d2, MASS ? smass[min(j + v, re - 1u)] : P.mass, P);
                const bool nb = j + v < re && d2 < P.hg2;
                rho = nb ? __fadd_rn(rho, w) : rho;
                // listed where the next neighbour overwrites it unless it counts (a branch costs more)
                nl[min(c_nb, kSmallList) * share + tid] = (uint16_t)(j + v);
                c_nb += nb && j + v != s ? 1u : 0u;  // j != i (fluid.rs:947-950)
              }
            }
          }
        }
        ncnt[tid] = c_nb;
        float dens = rho;
        if (dens < 0.0f) dens = 0.0f;
        if (dens > P.rho_cap) dens = P.rho_cap;
        const uint32_t ph = PHASE ? min((uint32_t)sphase[tid], 3u) : P.uniform_phase;
        const float p = eos(dens, P.rest[ph], P);
        const float rc = fmaxf(dens, kEps);
        const float2 dq = make_float2(dens, __fdiv_rn(p, __fmul_rn(rc, rc)));
        sdq[s] = dq;
        if (last) {
          A.sid[s] = sid[tid];
          A.sdq[s] = dq;
          A.spres[s] = p;
        }
      }
      cluster_sync();
      // ---- the window's densities from their owners
      for (uint32_t f = wlo + tid; f < whi; f += threads)
        if (f < first || f >= end) sdq[f] = load_remote(&sdq[f], f / share);
      __syncthreads();
      // ---- force + integrate (k_force_integrate / k_force_fast), kSmallLanes lanes per particle
      {
        constexpr uint32_t G = kSmallLanes, kRows = PLAIN ? 6u : 8u;
        const uint32_t gi = tid / G, l = tid % G, s = first + gi;
        const bool active = s < end;
        float* tb = terms + gi * kRows * G;
        float2 pi, vi, dqi;
        pi = vi = dqi = make_float2(0.0f, 0.0f);
        uint32_t total = 0u, ks = g.sentinel;
        float m_i = P.mass;
        if (active) {
          pi = spos[s], vi = svel[s], dqi = sdq[s];
          ks = skey[gi];
          total = ncnt[gi];
          if (MASS) m_i = smass[s];
        }
        const float rho_i = fmaxf(dqi.x, kEps), q_i = dqi.y;
        const uint32_t idle = active ? s : wlo;  // a slot for lanes without a pair
        FastPair fp;
        fp.pi = pi;
        fp.vi = vi;
        fp.rho_i = rho_i;
        fp.mq_i = __fmul_rn(P.mass, q_i);
        float acc = 0.0f;  // lanes 0, 1: the force sum's x, y; 2, 3: the XSPH sum's
        auto pairs = [&](uint32_t j, bool valid) {  // up to G pairs in visit order, lane l holds pair j
          if constexpr (FAST) {
            float2 nd, dv;
            float c, w;
            fp.terms(spos[j], svel[j], sdq[j], P, nd, c, dv, w);
            // a lane without a pair: all factors zero, also where the particle's own row is not finite
            tb[l] = valid ? nd.x : 0.0f;
            tb[G + l] = valid ? nd.y : 0.0f;
            tb[2u * G + l] = valid ? dv.x : 0.0f;
            tb[3u * G + l] = valid ? dv.y : 0.0f;
            tb[4u * G + l] = valid ? c : 0.0f;
            tb[5u * G + l] = valid ? w : 0.0f;
          } else {
            const PairTerms t =
                pair2_terms<PLAIN>(spos[j], svel[j], sdq[j], MASS ? smass[j] : P.mass, pi, vi, rho_i, q_i, m_i, P);
            tb[l] = valid ? t.nx : 0.0f;
            tb[G + l] = valid ? t.ny : 0.0f;
            tb[2u * G + l] = valid ? t.wx : 0.0f;
            tb[3u * G + l] = valid ? t.wy : 0.0f;
            if constexpr (!PLAIN) {
              tb[4u * G + l] = valid ? t.cx : 0.0f;
              tb[5u * G + l] = valid ? t.cy : 0.0f;
            }
          }
          __syncwarp();
          const float4 v = reinterpret_cast<const float4*>(tb)[l];
          if constexpr (FAST) {
            const float4 f = reinterpret_cast<const float4*>(tb)[l < 2u ? 4 : 5];
            acc = __fmaf_rn(v.x, f.x, acc);
            acc = __fmaf_rn(v.y, f.y, acc);
            acc = __fmaf_rn(v.z, f.z, acc);
            acc = __fmaf_rn(v.w, f.w, acc);
          } else if constexpr (PLAIN) {
            acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v.x), v.y), v.z), v.w);
          } else {
            float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (l < 2u) f = reinterpret_cast<const float4*>(tb)[4u + l];
            acc = __fadd_rn(__fadd_rn(acc, v.x), f.x);
            acc = __fadd_rn(__fadd_rn(acc, v.y), f.y);
            acc = __fadd_rn(__fadd_rn(acc, v.z), f.z);
            acc = __fadd_rn(__fadd_rn(acc, v.w), f.w);
          }
          __syncwarp();
        };
        if (!__any_sync(kAll, total > kSmallList)) {
          const uint32_t most_l = __reduce_max_sync(kAll, total);
#pragma unroll 1
          for (uint32_t o = l; o < most_l + l; o += G) {
            const bool valid = o < total;
            pairs(valid ? (uint32_t)nl[o * share + gi] : idle, valid);
          }
        } else {
          // a particle of the warp has more neighbours than its list holds:
          // the candidates of all, bucket by bucket
          const uint32_t bx = ks & g.maskw, by = ks >> g.log2w;
#pragma unroll 1
          for (uint32_t t = 0; t < 9u; t++) {
            uint32_t ws = 0u, we = 0u;
            if (ks != g.sentinel) {
              const uint32_t bb = (((by + t / 3u - 1u) & g.maskh) << g.log2w) + ((bx + t % 3u - 1u) & g.maskw);
              ws = start_of(bb);
              we = start_of(bb + 1u);
            }
            const uint32_t len = __reduce_max_sync(kAll, we - ws);
#pragma unroll 1
            for (uint32_t o = 0; o < len; o += G) {
              const uint32_t j = ws + o + l;
              bool nb = j < we && j != s;
              const uint32_t jj = nb ? j : idle;
              const float2 c = spos[jj];
              const float ex = __fsub_rn(c.x, pi.x), ey = __fsub_rn(c.y, pi.y);
              nb = nb && __fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)) < P.hg2;
              pairs(jj, nb);
            }
          }
        }
        const float fx = __shfl_sync(kAll, acc, 0, G), fy = __shfl_sync(kAll, acc, 1, G);
        float sx = __shfl_sync(kAll, acc, 2, G), sy = __shfl_sync(kAll, acc, 3, G);
        if constexpr (FAST) {
          const float xs = __fmul_rn(__fmul_rn(2.0f, P.mass), P.c_poly6);
          sx = __fmul_rn(sx, xs);
          sy = __fmul_rn(sy, xs);
        }
        const float ax = __fadd_rn(P.gx, __fdiv_rn(fx, rho_i));
        const float ay = __fadd_rn(P.gy, __fdiv_rn(fy, rho_i));
        if (active && l == 0u) {
          float4 out;
          integrate_state<false, true>(pi, vi, ax, ay, sx, sy, dt, P, s_bodies, out);
          const uint32_t id = sid[gi];
          const uint32_t nk = bucket_key(out.x, out.y, g);
          A.state[id] = out;
          A.key[id] = nk;
          if (last) atomicAdd(&A.count[nk], 1u);
        }
      }
      taken++;
      cluster_sync();  // the new states and keys; no block still reads this one's shared memory
    }
  }
  if (A.substeps && rank == 0u && tid == 0u) {
    const unsigned long long total = *A.substeps + taken;
    *A.substeps = total;
    *const_cast<volatile unsigned long long*>(A.substeps_host) = total;
  }
}
