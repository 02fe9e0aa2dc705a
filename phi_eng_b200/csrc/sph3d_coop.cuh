// Density and force passes with several threads per particle, included by
// sph3d.cu inside its anonymous namespace, for particle sets too small to fill
// the GPU with one thread each.
//
// One thread per particle walks ~216 candidates and ~33 pairs one after the
// other: on a 4,096-particle block 12.4 us (density) and 20.9 us (force) on 16
// and 32 of the 148 SMs, almost all of it one thread's latency. The density
// pass here gives each of a particle's nine candidate rows a thread of its own,
// the force pass gives each particle a group of eight lanes that evaluate its
// pairs side by side. Terms go through shared memory and are summed in the visit
// order, so every result has the bits of the one-thread passes; the row masks
// between the two passes are the same too.
constexpr uint32_t kRowTerms = 32;      // density terms kept per row
constexpr uint32_t kRowCount = 0xFFFFFFu;
constexpr uint32_t kCoopPairs = 128;    // listed neighbours of a group
constexpr uint32_t kCoopThreads = 256;  // block of the force pass
// Lanes per particle of the force pass: 8 and 32 differ by 5 % on 64 to 4,096
// particles (16.3 and 15.5 us per step, 29.1 and 28.4), and 32 waste lanes on
// more (8,000 particles: 32.6 against 36.1).
constexpr int kCoopLanes = 8;
// Largest particle sets that take these passes. Steps of 28^3, 36^3 and 40^3
// particles, density by rows against one thread per particle: 38.2 / 46.5,
// 46.7 / 49.3, 53.4 / 52.1 us (tolerance mode). Force by eight lanes against one
// thread, rows in both: exact 36.3 / 47.4, 52.2 / 56.3, 63.3 / 62.0; tolerance
// mode 36.6 / 38.2, 51.9 / 46.7, 63.8 / 53.4. Of compressed sets only those of
// several times the rest density are faster by one thread (0.2 apart at h 0.5 and
// 32,768 particles: 12 steps 1,254 us against 1,394 before these passes' last change,
// 0.12 apart 5,188 against 4,173).
constexpr uint32_t kRowsMax3 = 49152;
constexpr uint32_t kCoopMax3 = 49152, kCoopMaxFast3 = 24576;

// Density + EOS. Warp r of a block walks row r of the block's 32 particles,
// one per lane, and keeps the neighbours' terms; warp 0 then sums each
// particle's terms row by row. Of a row with more than kRowTerms neighbours
// warp 0 walks all but the first 32 slots itself (the particle's 27 cells anew:
// 32,768 particles 0.17 apart, h 0.5, 120 us instead of 48).
template <bool MASS, bool PHASE, bool WIDE>
__global__ void __launch_bounds__(288) k_density3_rows(const float4* __restrict__ spos,
                                                       const uint32_t* __restrict__ skey,
                                                       const float* __restrict__ smass,
                                                       const uint8_t* __restrict__ sphase, uint32_t n,
                                                       const uint32_t* __restrict__ start,
                                                       const uint32_t* __restrict__ sq, StepParams3 P,
                                                       float2* __restrict__ sdq, float* __restrict__ spres,
                                                       uint32_t* __restrict__ nmask) {
  chain_wait(spos, skey, smass, sphase, start, sq);
  __shared__ float terms[9][kRowTerms][32];
  __shared__ uint32_t row_cnt[9][32];  // kRowCount: neighbours; 24..29: those of m[0]; 30, 31: a second word, no masks
  const uint32_t p = threadIdx.x & 31u, r = threadIdx.x >> 5;
  const uint32_t s = blockIdx.x * 32u + p;
  const bool active = s < n;
  const GridPlan3& g = P.grid;
  const uint32_t k = active ? skey[s] : g.sentinel;
  const float4 pi = spos[active ? s : 0u];
  uint32_t cnt = 0, m[2] = {0u, 0u}, kind = 2u;
  if (k != g.sentinel) {
    const uint32_t bx = k & g.maskw, by = (k >> g.log2w) & g.maskh, bz = k >> (g.log2w + g.log2h);
    const uint32_t row = row_base3(by, bz, (int)r, g);
    const bool quick = quick_range(pi.x, pi.y, pi.z, P.cell_units);
    const uint32_t qi = sq[s];
    const bool seam = on_seam3(bx, g);
    const RowRange3 q = row_range3(row, bx, seam, g, start);
#pragma unroll 1
    for (uint32_t part = 0; part < (seam ? 2u : 1u); part++) {
      uint32_t found[2];
      const uint32_t rs = part ? q.rs2 : q.rs, re = part ? q.re2 : q.re;
      auto hit = [&](uint32_t j) {
        const float4 a = __ldg(&spos[j]);
        const float dx = __fsub_rn(a.x, pi.x), dy = __fsub_rn(a.y, pi.y), dz = __fsub_rn(a.z, pi.z);
        const float d2 = dot3(dx, dy, dz, dx, dy, dz);
        const bool nb = d2 < P.hg2;
        // kept where the next neighbour overwrites it unless it counts (a branch costs more)
        if (cnt < kRowTerms) terms[r][cnt][p] = __fmul_rn(MASS ? __ldg(&smass[j]) : P.mass, poly6_nb<WIDE>(d2, P));
        cnt += nb ? 1u : 0u;
        return nb;
      };
      row_candidates3(rs, re, qi, sq, found, hit, quick ? kQuickD2 : kEverySlot);
      if (part) m[1] = found[0];
      else m[0] = found[0], m[1] = found[1];
    }
    const uint32_t len = max(q.re - q.rs, q.re2 - q.rs2);
    kind = len > (seam ? 1u : 2u) * kMaskBits3 ? 2u : seam || len > kMaskBits3 ? 1u : 0u;
  }
  row_cnt[r][p] = cnt | (uint32_t)__popc(m[0]) << 24 | kind << 30;
  if (active) {
    nmask[(size_t)r * n + s] = m[0];
    if (kind == 1u) nmask[(size_t)(9u + r) * n + s] = m[1];
  }
  __syncthreads();
  if (r != 0u || !active) return;
  float rho = 0.0f;
  uint32_t flags = 0u;
  bool fits = true;
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const uint32_t kd = row_cnt[q][p] >> 30;
    flags |= kd == 0u ? 0u : kd == 1u ? 1u << q : kNoMasks;
    fits = fits && (row_cnt[q][p] & kRowCount) <= kRowTerms;
  }
  auto add_terms = [&](int q, uint32_t c) {
    for (uint32_t i = 0; i < c; i += 4) {
#pragma unroll
      for (uint32_t t = 0; t < 4; t++) {
        const float w = terms[q][i + t][p];
        rho = i + t < c ? __fadd_rn(rho, w) : rho;
      }
    }
  };
  if (fits) {
#pragma unroll
    for (int q = 0; q < 9; q++) add_terms(q, row_cnt[q][p] & kRowCount);
  } else {
    const uint32_t bx = k & g.maskw, by = (k >> g.log2w) & g.maskh, bz = k >> (g.log2w + g.log2h);
    const bool seam = on_seam3(bx, g);
#pragma unroll 1
    for (int q = 0; q < 9; q++) {
      const uint32_t c = row_cnt[q][p] & kRowCount;
      if (c <= kRowTerms) {
        add_terms(q, c);
        continue;
      }
      add_terms(q, row_cnt[q][p] >> 24 & 63u);  // those of the row's first 32 slots; then from there on
      const RowRange3 rr = row_range3(row_base3(by, bz, q, g), bx, seam, g, start);
#pragma unroll 1
      for (uint32_t part = 0; part < (seam ? 2u : 1u); part++) {
        const uint32_t e = part ? rr.re2 : rr.re;
#pragma unroll 8
        for (uint32_t j = part ? rr.rs2 : rr.rs + kMaskBits3; j < e; j++) {
          const float4 a = __ldg(&spos[j]);
          const float dx = __fsub_rn(a.x, pi.x), dy = __fsub_rn(a.y, pi.y), dz = __fsub_rn(a.z, pi.z);
          const float d2 = dot3(dx, dy, dz, dx, dy, dz);
          const float w = __fmul_rn(MASS ? __ldg(&smass[j]) : P.mass, poly6_nb<WIDE>(d2, P));
          rho = d2 < P.hg2 ? __fadd_rn(rho, w) : rho;
        }
      }
    }
  }
  nmask[18 * (size_t)n + s] = flags;
  float dens = rho;
  if (dens < 0.0f) dens = 0.0f;
  if (dens > P.rho_cap) dens = P.rho_cap;
  const uint32_t ph = PHASE ? min((uint32_t)sphase[s], 3u) : P.uniform_phase;
  const float pr = eos(dens, P.rest[ph], P);
  const float rc = fmaxf(dens, kEps);
  sdq[s] = make_float2(dens, __fdiv_rn(pr, __fmul_rn(rc, rc)));
  spres[s] = pr;
}

// Rows of the pair-term buffer of a group: exact mode na[3], xs[3] and, with
// the optional terms, co[3]; tolerance mode -d[3], dv[3], c, w (the factors of
// the fused multiply-adds).
template <bool MASS, bool DEBUG, bool PLAIN, bool FAST>
__global__ void __launch_bounds__(kCoopThreads) k_force3_coop(
    const float4* __restrict__ spos, const float4* __restrict__ svel, const float2* __restrict__ sdq,
    const uint32_t* __restrict__ skey, const uint32_t* __restrict__ sid, const float* __restrict__ smass, uint32_t n,
    const uint32_t* __restrict__ start, StepParams3 P, const DevBody3* __restrict__ bodies,
    const uint32_t* __restrict__ nmask, float4* __restrict__ pos_out,
    float4* __restrict__ vel_out, uint32_t* __restrict__ key_out, uint32_t* __restrict__ count_out,
    float4* __restrict__ dbg, uint32_t* __restrict__ pid) {
  chain_wait(spos, svel, sdq, skey, sid, smass, start, bodies, nmask);
  constexpr int G = kCoopLanes;
  static_assert(G == 8, "six lanes of a group hold the sums; lanes 0..7 expand rows 0..7");
  constexpr uint32_t kAll = 0xFFFFFFFFu, kGroups = kCoopThreads / G;
  constexpr int kRows = FAST ? 8 : PLAIN ? 6 : 9;
  constexpr uint32_t kStride = kRows * G + 4;  // a multiple of four floats: rows are read 16 bytes at a time
  __shared__ __align__(16) float tbuf_all[kGroups * kStride];
  __shared__ uint32_t list_all[kGroups * kCoopPairs];
  const uint32_t s0 = (blockIdx.x * kCoopThreads + threadIdx.x) / G;
  const uint32_t l = threadIdx.x % G;
  float* tbuf = tbuf_all + threadIdx.x / G * kStride;
  uint32_t* list = list_all + threadIdx.x / G * kCoopPairs;
  const bool active = s0 < n;
  const uint32_t s = active ? s0 : 0u;
  const uint32_t k = skey[s];
  const uint32_t id = sid[s];
  const float4 pi = spos[s];
  const float4 vi = svel[s];
  const float2 dqi = sdq[s];
  const float m_i = MASS ? smass[s] : P.mass;
  const float rho_i = fmaxf(dqi.x, kEps);
  const float q_i = dqi.y;
  const float mq_i = __fmul_rn(P.mass, q_i);
  const GridPlan3& g = P.grid;
  const uint32_t bx = k & g.maskw, by = (k >> g.log2w) & g.maskh, bz = k >> (g.log2w + g.log2h);
  const bool live = active && k != g.sentinel;
  const uint32_t flags = live ? nmask[18 * (size_t)n + s] : kNoMasks;
  bool listed = !(flags & kNoMasks);
  // the set bits of the nine rows' masks as one list of slots in visit order:
  // lane l expands row l, the first row 8 as well
  uint32_t mk[2] = {0u, 0u}, bs[2] = {0u, 0u}, mk8[2] = {0u, 0u}, bs8[2] = {0u, 0u};
  if (listed) {
    auto row_masks = [&](uint32_t r, uint32_t (&m)[2], uint32_t (&b)[2]) {
      const uint32_t row = row_base3(by, bz, (int)r, g);
      m[0] = nmask[(size_t)r * n + s];
      b[0] = row_first3(row, bx, g, start);
      if (flags >> r & 1u) {
        m[1] = nmask[(size_t)(9u + r) * n + s];
        b[1] = on_seam3(bx, g) ? __ldg(&start[row]) : b[0] + kMaskBits3;
      }
    };
    row_masks(l, mk, bs);
    if (l == 4u) {  // the particle's own bit: j != i (fluid3.rs:1041)
      if (s - bs[0] < kMaskBits3) mk[0] &= ~(1u << (s - bs[0]));
      else mk[1] &= ~(1u << (s - bs[1]));
    }
    if (l == 0u) row_masks(8u, mk8, bs8);
  }
  const uint32_t own = (uint32_t)(__popc(mk[0]) + __popc(mk[1]));
  uint32_t off = own;
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kAll, off, o, G);
    if (l >= (uint32_t)o) off += y;
  }
  uint32_t cnt = __shfl_sync(kAll, off, 7, G);
  const uint32_t off8 = cnt;
  cnt += (uint32_t)__shfl_sync(kAll, __popc(mk8[0]) + __popc(mk8[1]), 0, G);
  if (cnt > kCoopPairs) listed = false;
  if (listed) {
    off -= own;
#pragma unroll
    for (int h = 0; h < 2; h++)
      for (; mk[h]; mk[h] &= mk[h] - 1u) list[off++] = bs[h] + (uint32_t)(__ffs((int)mk[h]) - 1);
    off = off8;
#pragma unroll
    for (int h = 0; h < 2; h++)
      for (; mk8[h]; mk8[h] &= mk8[h] - 1u) list[off++] = bs8[h] + (uint32_t)(__ffs((int)mk8[h]) - 1);
  }
  __syncwarp();
  float acc = 0.0f;  // lanes 0..2: the force sum's x, y, z; 3..5: the XSPH sum's
  auto chunk = [&](uint32_t j, bool valid) {  // up to G pairs in visit order, lane l holds pair j
    if constexpr (FAST) {
      float nd[3] = {0.0f, 0.0f, 0.0f}, dv[3] = {0.0f, 0.0f, 0.0f}, c = 0.0f, w = 0.0f;
      if (valid) pair3_fast_terms(j, pi, vi, rho_i, mq_i, spos, svel, sdq, P, nd, dv, c, w);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        tbuf[a * G + l] = nd[a];
        tbuf[(3 + a) * G + l] = dv[a];
      }
      tbuf[6 * G + l] = c;
      tbuf[7 * G + l] = w;
    } else {
      float na[3] = {0.0f, 0.0f, 0.0f}, co[3] = {0.0f, 0.0f, 0.0f}, xs[3] = {0.0f, 0.0f, 0.0f};
      if (valid) pair3_terms<MASS, PLAIN>(j, pi, vi, rho_i, q_i, m_i, spos, svel, sdq, smass, P, na, co, xs);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        tbuf[a * G + l] = na[a];
        tbuf[(3 + a) * G + l] = xs[a];
        if constexpr (!PLAIN) tbuf[(6 + a) * G + l] = co[a];
      }
    }
    __syncwarp();
    if (l < 6u) {
      const float4* row = reinterpret_cast<const float4*>(tbuf + l * G);
#pragma unroll
      for (int q = 0; q < G / 4; q++) {
        const float4 a = row[q];
        if constexpr (FAST) {
          const float4 b = reinterpret_cast<const float4*>(tbuf + (l < 3u ? 6 : 7) * G)[q];
          acc = __fmaf_rn(a.x, b.x, acc);
          acc = __fmaf_rn(a.y, b.y, acc);
          acc = __fmaf_rn(a.z, b.z, acc);
          acc = __fmaf_rn(a.w, b.w, acc);
        } else if constexpr (PLAIN) {
          acc = __fadd_rn(acc, a.x);
          acc = __fadd_rn(acc, a.y);
          acc = __fadd_rn(acc, a.z);
          acc = __fadd_rn(acc, a.w);
        } else {
          const float4 b = l < 3u ? reinterpret_cast<const float4*>(tbuf + (6 + l) * G)[q]
                                  : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          acc = __fadd_rn(__fadd_rn(acc, a.x), b.x);
          acc = __fadd_rn(__fadd_rn(acc, a.y), b.y);
          acc = __fadd_rn(__fadd_rn(acc, a.z), b.z);
          acc = __fadd_rn(__fadd_rn(acc, a.w), b.w);
        }
      }
    }
    __syncwarp();
  };
  const uint32_t most = __reduce_max_sync(kAll, listed ? cnt : 0u);
  for (uint32_t o = 0; o < most; o += G) {
    const bool in = listed && o + l < cnt;
    chunk(in ? list[o + l] : s, in);
  }
  const bool walk = live && !listed;
  if (__any_sync(kAll, walk)) {
    // no masks (a row too long for them) or a full list: the
    // candidates, bucket by bucket
#pragma unroll 1
    for (int t = 0; t < 27; t++) {
      uint32_t rs = 0u, re = 0u;
      if (walk) {
        const uint32_t b = row_base3(by, bz, t / 3, g) | ((bx + (uint32_t)(t % 3) - 1u) & g.maskw);
        rs = __ldg(&start[b]);
        re = __ldg(&start[b + 1]);
      }
      const uint32_t len = __reduce_max_sync(kAll, re - rs);
      for (uint32_t o = 0; o < len; o += G) {
        const uint32_t j = rs + o + l;
        bool nb = j < re && j != s;
        if (nb) {
          const float4 a = __ldg(&spos[j]);
          const float ex = __fsub_rn(a.x, pi.x), ey = __fsub_rn(a.y, pi.y), ez = __fsub_rn(a.z, pi.z);
          nb = dot3(ex, ey, ez, ex, ey, ez) < P.hg2;
        }
        chunk(j, nb);
      }
    }
  }
  float f[3], sm[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    f[a] = __shfl_sync(kAll, acc, a, G);
    sm[a] = __shfl_sync(kAll, acc, 3 + a, G);
  }
  if (!active) return;
  finish3<DEBUG, PLAIN, FAST>(s, id, pid, l == 0u, pi, vi, rho_i, q_i, f, sm, P, bodies, pos_out, vel_out, key_out,
                              count_out, dbg);
}
