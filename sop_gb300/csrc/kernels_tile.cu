// The steps of small contexts, with everything the force sum reads staged in
// shared memory by asynchronous copies: over tiles of 16 or 32 consecutive
// beads a block (k_step_tile, from tables k_pl_tile builds at each pair-list
// rebuild), or with the pair-list rebuild in the same launch (k_pair_step).
//
// k_pl_tile writes per tile what the steps until the next rebuild need and
// nothing else:
//   - the distinct beads the tile's force sums touch (its own and every
//     partner), ascending, so a step reads each coordinate once per tile instead
//     of once per pair;
//   - the repulsive rows as indices into that list, and the bonded, angle and
//     native entries as {r0, eps, index, type}, in the order the lanes take them.
// k_step_tile then copies the rows (which no step changes: they are on their
// way before the previous step has finished, under programmatic dependent
// launch, and so is the bead's noise) and, after it, the listed coordinates and
// the beads' state, and does the rest from shared memory.
//
// What bounds k_step (kernels_step.cu) in a small context is latency: a chain
// of about seven reads from L2 per bead and step, 8 us a step from 128 to 4,000
// beads.  Here one round trip to L2 lies between the steps.  us of a run and a
// read of the state with k_step / staged, list rebuilds included: 100 steps of 128
// beads 599 / 472, of 4,000 beads 884 / 788, extended 640 / 544; 50 steps of 1,531
// beads with a list before every step 667 / 505.
//
// The per-entry and per-bead arithmetic is k_step's (step_dev.cuh) in the same
// order, so every bit is the same.  A tile whose lists do not fit (long rows, a
// dense structure) gathers as k_step does.
#include <algorithm>
#include <type_traits>

#include "lists_dev.cuh"
#include "step_force.cuh"

namespace sop {

// ------------------------------------------------------------- async copies
__device__ __forceinline__ void copy16(void* shared, const void* global) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(shared);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(global) : "memory");
}
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Entries of bead q's repulsive row in a tile's table: chunks of 16, four
// words of four entries each (word w: entries w, w + 4, w + 8, w + 12, what one
// lane of four sums), the words of the tile's beads side by side.
template <int TB>
__device__ __forceinline__ int tile_rep_at(int q, int e) {
  return ((((e >> 4) * 4 + (e & 3)) * TB + q) << 2) + ((e >> 2) & 3);
}

// ------------------------------------------------------------------- build
constexpr int kTileThreads = 256;

// The pair-list rebuild of a tile's beads (a warp per bead, as k_pl) and the
// tile's tables from it, one block per tile: as launches of their own the two
// took 11 + 16 us at 4,000 beads.
constexpr int kBuildThreads = 512;
template <int TB, bool UNI>
__global__ void __launch_bounds__(kBuildThreads) k_pl_tile(DevSys s, TileSet ts, int koff, int only_tables) {
  constexpr int kWarps = kBuildThreads / 32;
  __shared__ unsigned bits[kTileWords];
  __shared__ unsigned short pre[kTileWords];
  __shared__ int warp_sum[kWarps];
  __shared__ int most_rep, most_small;
  __shared__ int2 rows[TB];  // lengths: repulsive, attractive
  pdl_wait();
  pdl_release();
  if (*s.flags & FLAG_NL_OVERFLOW) return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, tile = blockIdx.x;
  const int b0 = tile * TB, nb = min(TB, s.nlive - b0);
  const MolConst& mf = s.mol[s.mol_of[b0]];
  const MolConst& ml = s.mol[s.mol_of[b0 + nb - 1]];
  const int lo = mf.start, words = (ml.start + ml.n - lo + 31) >> 5;
  const bool fits = words <= kTileWords;  // the same for every thread
  if (t == 0) most_rep = most_small = 0;
  if (fits)
    for (int w = t; w < words; w += kBuildThreads) bits[w] = 0;
  __syncthreads();
  auto mark = [&](int j) {
    if (fits) atomicOr(bits + ((j - lo) >> 5), 1u << ((j - lo) & 31));
  };
  for (int q = warp; q < nb; q += kWarps) {
    const int i = b0 + q, m = s.mol_of[i], start = s.mol[m].start;
    const int2 br = s.bond_row[i], ar = s.ang_row[i];
    int nrep, natt;
    if (!only_tables && mol_listed(s, m, koff)) {
      pair_rows<UNI, 32, false>(
          s, xbuf(s, m, koff), i, pair_head<32, false>(s, i, m), [&](int, int j) { mark(start + j); },
          [&](int, float4 a) { mark(__float_as_int(a.x)); }, nrep, natt);
    } else {  // the rows stay as they are
      nrep = s.pl_cnt[i];
      natt = s.pl_att_cnt[i];
      for (int e = lane; e < nrep; e += 32) mark(start + (int)s.pl_j[(long long)i * s.nl_stride + pl_at(e)]);
      for (int e = lane; e < natt; e += 32) mark(__float_as_int(s.pl_att[s.nat_row[i].x + e].x));
    }
    for (int e = lane; e < br.y; e += 32) mark(s.bond_j[br.x + e]);
    for (int e = lane; e < ar.y; e += 32) mark(s.ang_j[ar.x + e]);
    if (lane == 0) {
      mark(i);
      rows[q] = make_int2(nrep, natt);
      atomicMax(&most_rep, nrep);
      atomicMax(&most_small, br.y + ar.y + natt);
    }
  }
  __syncthreads();
  // exclusive prefix of the words' bit counts, a run of words per thread
  const int per = fits ? (words + kBuildThreads - 1) / kBuildThreads : 0;
  const int w0 = min(t * per, words), w1 = min(w0 + per, words);
  int sum = 0;
  for (int w = w0; w < w1; ++w) sum += __popc(bits[w]);
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int at = incl - sum, total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) at += warp_sum[w];
    total += warp_sum[w];
  }
  const int chunks = (most_rep + 15) >> 4, small = most_small;
  if (!fits || total > kTileCap || chunks > kTileChunks || small > kTileSmall ||
      tile_smem(TB, total, chunks, small) > ts.smem) {
    if (t == 0) ts.cnt[tile] = -1;
    return;
  }
  int* list = ts.bead + (long long)tile * kTileCap;
  for (int w = w0; w < w1; ++w) {
    pre[w] = (unsigned short)at;
    for (unsigned m = bits[w]; m; m &= m - 1) list[at++] = lo + 32 * w + __ffs(m) - 1;
  }
  __syncthreads();
  auto local = [&](int j) {
    const int w = (j - lo) >> 5;
    return (int)pre[w] + __popc(bits[w] & ((1u << ((j - lo) & 31)) - 1u));
  };
  if (t == 0) {
    ts.cnt[tile] = total;
    ts.dim[tile] = make_int2(chunks | (small << 16), local(b0));
  }
  unsigned short* rep = ts.rep + (long long)tile * kTileChunks * 16 * TB;
  for (int q = warp; q < nb; q += kWarps) {
    const int i = b0 + q, start = s.mol[s.mol_of[i]].start;
    const int2 br = s.bond_row[i], ar = s.ang_row[i];
    const int nat0 = s.nat_row[i].x, nrep = rows[q].x, nba = br.y + ar.y, nsmall = nba + rows[q].y;
    const int own = (nrep + 15) >> 4, self = local(i);
    if (lane == 0) ts.num[i] = nsmall | (own << 16);
    const unsigned short* row = s.pl_j + (long long)i * s.nl_stride;
    // past the row's end the partner is the bead itself (d2 = 0 contributes 0)
    for (int e = lane; e < 16 * own; e += 32)
      rep[tile_rep_at<TB>(q, e)] = (unsigned short)(e < nrep ? local(start + (int)row[pl_at(e)]) : self);
    float4* out = ts.small + (long long)tile * kTileSmall * TB + q;
    for (int e = lane; e < nsmall; e += 32) {
      float4 a = make_float4(0.f, 0.f, 0.f, __int_as_float(1));  // {r0, eps, position, type}
      int j;
      if (e < br.y) {
        j = s.bond_j[br.x + e];
        a.x = s.bond_r0[br.x + e];
        a.w = __int_as_float(0);
      } else if (e < nba) {
        j = s.ang_j[ar.x + e - br.y];
      } else {
        const float4 c = s.pl_att[nat0 + e - nba];
        j = __float_as_int(c.x);
        a.x = c.y;
        a.y = c.z;
        a.w = __int_as_float(2);
      }
      a.z = __int_as_float(local(j));
      out[e * TB] = a;
    }
  }
}

// -------------------------------------------------------------------- step
// The force on a tile's bead from the staged tables, G lanes a bead: lane
// `lane` of G sums virtual lanes lane + c * G (the order of bead_force).
template <int TB, bool UNI, bool wrap_list>
__device__ __forceinline__ void tile_force(const DevSys& s, const float4* x, const float4* small,
                                           const unsigned short* rep, bool wrap, int q, int self, int nsmall,
                                           int chunks, int lane, float& fx, float& fy, float& fz,
                                           bool& fene_bad) {
  constexpr int G = kTileThreads / TB, kC = kV / G;
  float ax[kC], ay[kC], az[kC];
#pragma unroll
  for (int c = 0; c < kC; ++c) ax[c] = ay[c] = az[c] = 0.f;
  const float4 xi = x[self];
  for (int base = 0; base < nsmall; base += kV) {
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      const int e = base + lane + c * G;
      if (e >= nsmall) continue;
      const float4 a = small[e * TB + q];
      const float4 xj = x[__float_as_int(a.z)];
      float lx, ly, lz;
      float dx = diff_exact(xj.x, xi.x, lx), dy = diff_exact(xj.y, xi.y, ly),
            dz = diff_exact(xj.z, xi.z, lz);
      if (wrap) min_image3(dx, dy, dz, s.boxl);
      const float cc =
          small_coeff(s, __float_as_int(a.w), dx, dy, dz, lx, ly, lz, a.x, a.y, fene_bad);
      acc3(ax[c], ay[c], az[c], cc, dx, dy, dz);
    }
  }
  const RepConst rc = rep_const(s);
  for (int t = 0; t < chunks; ++t) {
    int j[kC];
    if (G == 4) {
      const uint2 w = *reinterpret_cast<const uint2*>(rep + ((t * 4 + lane) * TB + q) * 4);
      j[0] = (int)(w.x & 0xffffu);
      j[1 % kC] = (int)(w.x >> 16);
      j[2 % kC] = (int)(w.y & 0xffffu);
      j[3 % kC] = (int)(w.y >> 16);
    } else {
      const unsigned short* w = rep + ((t * 4 + (lane & 3)) * TB + q) * 4 + (lane >> 2);
#pragma unroll
      for (int c = 0; c < kC; ++c) j[c] = (int)w[2 * c];
    }
    float4 xx[kC];
#pragma unroll
    for (int c = 0; c < kC; ++c) xx[c] = x[j[c]];
#pragma unroll
    for (int c = 0; c < kC; ++c) rep_entry<UNI, wrap_list>(rc, xi, xx[c], ax[c], ay[c], az[c]);
  }
  group_sum<G>(ax, ay, az, fx, fy, fz, fene_bad);
}

// Completes bead b from its force sum and its staged state and noise.
__device__ __forceinline__ void finish_staged(const DevSys& s, int b, int m, int koff, float4 fs,
                                              float4 inc, float4 p, float4 x, float3 z) {
  if (__float_as_int(fs.w) == 0) return;  // not stepped
  BeadState st;
  st.mc = s.mol[m];
  st.nb = s.mol_step[m] + 1 + koff;
  st.inc = inc;
  st.pi = p;
  st.xo = x;
  // the velocity is read only where the step keeps it
  st.vi = (st.nb <= 0 || st.mc.t_zero) ? s.v[b] : make_float4(0.f, 0.f, 0.f, 0.f);
  st.z = z;
  complete_bead<true>(s, b, m, fs, (int)(st.nb & 1), st);
}

// Step mol_step + 1 + koff of every bead.  early: the kernel before this one
// on the stream is a step too, so all a step does not write (the tables, the
// molecules' constants and clocks) is read before that one has finished.
template <int TB, bool UNI>
__global__ void __launch_bounds__(kTileThreads, 4) k_step_tile(DevSys s, TileSet ts, int koff, int early) {
  constexpr int G = kTileThreads / TB;
  extern __shared__ float4 dyn[];
  __shared__ float4 fsum[TB];
  __shared__ float4 inc0[TB], p0[TB];
  __shared__ float3 z[TB];
  const int t = threadIdx.x, tile = blockIdx.x;
  const int b0 = tile * TB, nb = min(TB, s.nlive - b0);
  const int q = t / G, lane = t % G;
  if (!early) pdl_wait();
  const bool frozen = *s.flags & FLAG_NL_OVERFLOW;
  const int cnt = ts.cnt[tile];
  const int2 dim = ts.dim[tile];
  const int chunks = dim.x & 0xffff, small = dim.x >> 16;
  float4* const stable = dyn + max(cnt, 0);
  uint4* const rtable = reinterpret_cast<uint4*>(stable + small * TB);
  int num = 0, m = 0;
  long long n = 0;
  bool run = false, wrap = false, wrap_list = false;
  if (q < nb) {
    m = s.mol_of[b0 + q];
    num = ts.num[b0 + q];
    const MolConst& mc = s.mol[m];
    n = s.mol_step[m] + 1 + koff;
    run = mc.active && n >= 0 && !(mc.nsteps >= 0 && n > mc.nsteps) && !frozen;
  }
  // a listed bead's coordinates at its own molecule's step
  auto source = [&](int b) {
    const long long step = s.mol_step[s.mol_of[b]] + 1 + koff;
    return s.x[(int)(step & 1)] + b;
  };
  constexpr int kAhead = 4;  // listed beads per thread whose addresses are found early
  const float4* from[kAhead];
  const int* list = ts.bead + (long long)tile * kTileCap;
#pragma unroll
  for (int k = 0; k < kAhead; ++k) {
    const int l = t + k * kTileThreads;
    from[k] = l < cnt ? source(list[l]) : nullptr;
  }
  if (cnt > 0) {
    const float4* st = ts.small + (long long)tile * kTileSmall * TB;
    for (int k = t; k < small * TB; k += kTileThreads) copy16(stable + k, st + k);
    const uint4* rt = reinterpret_cast<const uint4*>(ts.rep + (long long)tile * kTileChunks * 16 * TB);
    for (int k = t; k < chunks * 2 * TB; k += kTileThreads) copy16(rtable + k, rt + k);
  }
  int m2 = 0;  // of bead b0 + t, which thread t < nb completes
  if (t < nb) {
    m2 = s.mol_of[b0 + t];
    const MolConst& mc = s.mol[m2];
    z[t] = bead_noise(s, b0 + t, mc.start, s.mol_step[m2] + 1 + koff, mc.traj);
  }
  if (early) pdl_wait();
  pdl_release();
  if (run) {  // a step may set these
    run = s.mol_status[m] == 0;
    wrap = s.grid[m].wrap != 0;
    wrap_list = list_image_taken(s, m, n);
  }
  if (t < nb) {
    const long long n2 = s.mol_step[m2] + 1 + koff;
    copy16(inc0 + t, s.incr + b0 + t);
    copy16(p0 + t, s.p[(int)(n2 & 1)] + b0 + t);
  }
#pragma unroll
  for (int k = 0; k < kAhead; ++k)
    if (from[k]) copy16(dyn + t + k * kTileThreads, from[k]);
  for (int l = t + kAhead * kTileThreads; l < cnt; l += kTileThreads) copy16(dyn + l, source(list[l]));
  copies_done();
  __syncthreads();
  float fx = 0.f, fy = 0.f, fz = 0.f;
  bool bad = false;
  if (run) {
    if (cnt >= 0) {
      const unsigned short* rep = reinterpret_cast<const unsigned short*>(rtable);
      if (wrap_list)
        tile_force<TB, UNI, true>(s, dyn, stable, rep, wrap, q, dim.y + q, num & 0xffff, num >> 16, lane,
                                  fx, fy, fz, bad);
      else
        tile_force<TB, UNI, false>(s, dyn, stable, rep, wrap, q, dim.y + q, num & 0xffff, num >> 16, lane,
                                   fx, fy, fz, bad);
    } else {
      const int i = b0 + q;
      const int2 br = s.bond_row[i], ar = s.ang_row[i];
      bead_force<G, UNI>(s, GlobalX{s.x[(int)(n & 1)]}, i, m, n, lane, br, ar, s.nat_row[i].x,
                         s.pl_att_cnt[i], s.pl_cnt[i], fx, fy, fz, bad);
    }
  }
  if (lane == 0 && q < nb)
    fsum[q] = run ? marked_sum(fx, fy, fz, bad, n) : make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  if (t >= nb) return;
  finish_staged(s, b0 + t, m2, koff, fsum[t], inc0[t], p0[t],
                cnt >= 0 ? dyn[dim.y + t] : s.x[(int)((s.mol_step[m2] + 1 + koff) & 1)][b0 + t], z[t]);
}

// ----------------------------------------- pair list before every step
// A pair-list rebuild and the step after it in one launch, 16 or 8 lanes a bead: the
// group filters the bead's neighbour-list row by the last step's coordinates
// (pair_rows), keeps the surviving entries in shared memory, and sums the force
// over them at the step's own.  The step writes its look-ahead over the last
// step's coordinates while other blocks still filter by them, so those are kept
// a second time (s.xl, each step's in the buffer of its parity).  For contexts that rebuild the pair list before
// every step (the reference's cadence), where the two launches and the rows'
// way through L2 took 16 us a step at 1,531 beads.
// A block's molecules (from its first bead's to its last bead's) are staged in
// shared memory where they fit in `win` beads, else gathered from L2.
constexpr int kPairWindow = 1600; // most staged beads (two sets: 51 KB, three blocks of 16 lanes an SM)
constexpr int kPairRep = 256;     // entries of a repulsive row kept in shared memory
constexpr int kPairAtt = 32;      // and of an attractive one (past them: read from L2)
template <int G, bool UNI>
__global__ void __launch_bounds__(kTileThreads, 4) k_pair_step(DevSys s, int koff, int early, int win) {
  constexpr int kPairBeads = kTileThreads / G, kC = kV / G;
  extern __shared__ float4 dyn[];  // staged coordinates: the step's, then the last one's
  __shared__ unsigned short rrow[kPairBeads][kPairRep];
  __shared__ float4 arow[kPairBeads][kPairAtt];
  __shared__ float4 fsum[kPairBeads], inc0[kPairBeads], p0[kPairBeads], x0[kPairBeads];
  __shared__ float3 z[kPairBeads];
  const int t = threadIdx.x, q = t / G, lane = t % G;
  const int b0 = blockIdx.x * kPairBeads, nb = min(kPairBeads, s.nlive - b0), i = b0 + q;
  if (!early) pdl_wait();
  const bool frozen = *s.flags & FLAG_NL_OVERFLOW;
  const int mf = s.mol_of[b0], ml = s.mol_of[b0 + nb - 1];
  const int lo = s.mol[mf].start, range = s.mol[ml].start + s.mol[ml].n - lo;
  const int par = (int)((s.mol_step[mf] + 1 + koff) & 1);  // the step's buffer
  int m = 0;
  long long n = 0;
  bool run = false, other = false;
  int2 br = make_int2(0, 0), ar = br;
  int j0 = 0;  // the lane's bonded or angle entry
  float r0 = 0.f;
  PairHead head = {};
  if (q < nb) {
    m = s.mol_of[i];
    const MolConst& mc = s.mol[m];
    n = s.mol_step[m] + 1 + koff;
    run = mc.active && n >= 0 && !(mc.nsteps >= 0 && n > mc.nsteps) && !frozen;
    other = (int)(n & 1) != par;
    br = s.bond_row[i];
    ar = s.ang_row[i];
    head = pair_head<G, true>(s, i, m);
    if (lane < br.y) {
      j0 = s.bond_j[br.x + lane];
      r0 = s.bond_r0[br.x + lane];
    } else if (lane < br.y + ar.y) {
      j0 = s.ang_j[ar.x + lane - br.y];
    }
  }
  // staged: the block's molecules fit, all at steps of one parity
  const bool stage = !__syncthreads_or(other) && range <= win;
  int m2 = 0;
  if (t < nb) {
    m2 = s.mol_of[b0 + t];
    const MolConst& mc = s.mol[m2];
    z[t] = bead_noise(s, b0 + t, mc.start, s.mol_step[m2] + 1 + koff, mc.traj);
  }
  if (early) pdl_wait();
  pdl_release();
  if (stage)
    for (int l = t; l < range; l += kTileThreads) {
      copy16(dyn + win + l, s.xl[par ^ 1] + lo + l);
      copy16(dyn + l, s.x[par] + lo + l);
    }
  if (run) {  // a step may set these
    run = s.mol_status[m] == 0;
    head.wrap = s.grid[m].wrap != 0;
    head.wrap_list = list_image_taken(s, m, n);
  }
  if (t < nb) {
    const int cur = (int)((s.mol_step[m2] + 1 + koff) & 1);
    copy16(inc0 + t, s.incr + b0 + t);
    copy16(p0 + t, s.p[cur] + b0 + t);
    copy16(x0 + t, s.x[cur] + b0 + t);
  }
  copies_done();
  __syncthreads();
  float fx = 0.f, fy = 0.f, fz = 0.f;
  bool bad = false;
  // the bead's rows by the last step's coordinates XL, its force at the step's X
  auto bead = [&](const float4* XL, const float4* X) {
    int nrep, natt;
    pair_rows<UNI, G, true>(
        s, XL, i, head,
        [&](int pos, int j) {
          if (pos < kPairRep) rrow[q][pos] = (unsigned short)j;
        },
        [&](int pos, float4 a) {
          if (pos < kPairAtt) arow[q][pos] = a;
        },
        nrep, natt);
    __syncwarp(group_mask<G>(t & 31));
    const int start = head.mstart;
    const unsigned short* grow = s.pl_j + (long long)i * s.nl_stride;
    const float4 xi = X[i];
    const RepConst rc = rep_const(s);
    float ax[kC] = {}, ay[kC] = {}, az[kC] = {};
    const int nba = br.y + ar.y, nsmall = nba + natt;
    auto sum = [&](auto wrapped) {
      constexpr bool wrap_list = decltype(wrapped)::value;
      for (int base = 0; base < nsmall; base += kV) {
#pragma unroll
        for (int c = 0; c < kC; ++c) {
          const int e = base + lane + c * G;
          if (e >= nsmall) continue;
          int j = j0, type = e < br.y ? 0 : e < nba ? 1 : 2;
          float r = r0, eps = 0.f;
          if (type == 2) {
            const float4 a = e - nba < kPairAtt ? arow[q][e - nba] : s.pl_att[head.row.x + e - nba];
            j = __float_as_int(a.x);
            r = a.y;
            eps = a.z;
          } else if (e >= G) {
            j = type == 0 ? s.bond_j[br.x + e] : s.ang_j[ar.x + e - br.y];
            r = type == 0 ? s.bond_r0[br.x + e] : 0.f;
          }
          const float4 xj = X[j];
          float lx, ly, lz;
          float dx = diff_exact(xj.x, xi.x, lx), dy = diff_exact(xj.y, xi.y, ly),
                dz = diff_exact(xj.z, xi.z, lz);
          if (head.wrap) min_image3(dx, dy, dz, s.boxl);
          const float cc = small_coeff(s, type, dx, dy, dz, lx, ly, lz, r, eps, bad);
          acc3(ax[c], ay[c], az[c], cc, dx, dy, dz);
        }
      }
      constexpr int kB = 4;  // gathers in flight: kB / kC chunks
      for (int e0 = lane; e0 < nrep; e0 += kB * G) {
        float4 xx[kB];
#pragma unroll
        for (int c = 0; c < kB; ++c) {
          const int e = e0 + c * G;
          xx[c] = e < nrep ? X[start + (int)(e < kPairRep ? rrow[q][e] : grow[pl_at(e)])] : xi;
        }
#pragma unroll
        for (int c = 0; c < kB; ++c)  // past the row's end: the bead itself contributes 0
          rep_entry<UNI, wrap_list>(rc, xi, xx[c], ax[c % kC], ay[c % kC], az[c % kC]);
      }
    };
    if (head.wrap_list) sum(std::true_type{});
    else sum(std::false_type{});
    group_sum<G>(ax, ay, az, fx, fy, fz, bad);
  };
  if (run) {
    if (stage) bead(dyn + win - lo, dyn - lo);
    else bead(s.xl[(int)((n + 1) & 1)], s.x[(int)(n & 1)]);
  }
  if (lane == 0 && q < nb)
    fsum[q] = run ? marked_sum(fx, fy, fz, bad, n) : make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  if (t >= nb || __float_as_int(fsum[t].w) == 0) return;
  s.xl[(int)((s.mol_step[m2] + 1 + koff) & 1)][b0 + t] = x0[t];
  finish_staged(s, b0 + t, m2, koff, fsum[t], inc0[t], p0[t], x0[t], z[t]);
}

// ---------------------------------------------------------------- launchers
template <int TB>
static cudaError_t step_tb(const DevSys& s, const TileSet& ts, int koff, bool early, cudaStream_t st) {
  auto kernel = s.uniform_type ? k_step_tile<TB, true> : k_step_tile<TB, false>;
  // a per-kernel ceiling, always the same value
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             kTileSmemMost);
  if (e != cudaSuccess) return e;
  return launch_pdl_smem(kernel, (unsigned)ts.ntile, kTileThreads, (size_t)ts.smem, st, s, ts, koff,
                         early ? 1 : 0);
}

cudaError_t launch_step_tile(const DevSys& s, const TileSet& ts, int koff, bool early,
                             cudaStream_t st) {
  return ts.beads == 16 ? step_tb<16>(s, ts, koff, early, st) : step_tb<32>(s, ts, koff, early, st);
}

// The pair-list rebuild of s's molecules and the tables of every tile
// (only_tables: the lists stay as they are).
template <int TB>
static cudaError_t pl_tb(const DevSys& s, const TileSet& ts, int koff, bool only_tables, cudaStream_t st) {
  return launch_pdl(s.uniform_type ? k_pl_tile<TB, true> : k_pl_tile<TB, false>, (unsigned)ts.ntile,
                    kBuildThreads, st, s, ts, koff, only_tables ? 1 : 0);
}

cudaError_t launch_pl_tile(const DevSys& s, const TileSet& ts, int koff, bool only_tables,
                           cudaStream_t st) {
  return ts.beads == 16 ? pl_tb<16>(s, ts, koff, only_tables, st)
                        : pl_tb<32>(s, ts, koff, only_tables, st);
}

// The pair-list rebuild and the step after it, 8 or 16 lanes a bead.
template <int G>
static auto pair_kernel(const DevSys& s) { return s.uniform_type ? k_pair_step<G, true> : k_pair_step<G, false>; }

static size_t pair_smem(int win) { return 2 * (size_t)win * sizeof(float4); }

template <int G>
static cudaError_t pair_g(const DevSys& s, int koff, bool early, int win, cudaStream_t st) {
  auto kernel = pair_kernel<G>(s);
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)pair_smem(kPairWindow));
  if (e != cudaSuccess) return e;
  constexpr int beads = kTileThreads / G;
  return launch_pdl_smem(kernel, (unsigned)((s.nlive + beads - 1) / beads), kTileThreads, pair_smem(win), st,
                         s, koff, early ? 1 : 0, win);
}

cudaError_t launch_pair_step(const DevSys& s, const PairPlan& p, int koff, bool early, cudaStream_t st) {
  return p.lanes == 16 ? pair_g<16>(s, koff, early, p.win, st) : pair_g<8>(s, koff, early, p.win, st);
}

// The window takes shared memory, so fewer blocks are resident: it is used
// where the context's blocks run in as many waves with it as without.  us per 50
// steps with the window / without, factor cut-offs: one molecule of 800 beads 313 /
// 344, 1,531 350 / 359, 10 of 400 343 / 352, at 32 A 6 of 1,200 655 / 782 and (two
// waves both) 8 of 1,500 1,137 / 1,167; where it takes a wave more 5 of 1,600 729 /
// 480, 20 of 800 797 / 605, 13 of 1,495 956 / 672, at 32 A 5 of 1,500 874 / 820.
template <int G>
static cudaError_t plan_g(const DevSys& s, int max_mol, PairPlan* p) {
  auto kernel = pair_kernel<G>(s);
  int dev = 0, sms = 0, with = 0, without = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pair_smem(kPairWindow));
  const int win = max_mol > kPairWindow ? 0 : (max_mol + 256 < kPairWindow ? max_mol + 256 : kPairWindow);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&with, kernel, kTileThreads, pair_smem(win));
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&without, kernel, kTileThreads, 0);
  if (e != cudaSuccess) return e;
  constexpr int beads = kTileThreads / G;
  const long long blocks = (s.nlive + beads - 1) / beads;
  auto waves = [&](int resident) { return (blocks - 1) / std::max(1LL, (long long)resident * sms); };
  p->lanes = G;
  p->win = waves(with) <= waves(without) ? win : 0;
  p->wave = (long long)without * sms * beads;
  return cudaSuccess;
}

cudaError_t plan_pair_step(const DevSys& s, int lanes, int max_mol, PairPlan* p) {
  return lanes == 16 ? plan_g<16>(s, max_mol, p) : plan_g<8>(s, max_mol, p);
}

}  // namespace sop
