// The force sum of a bead over its rows, gathering partners by bead index.
#pragma once
#include "step_dev.cuh"

namespace sop {

// Coordinate sources of the force sum: the molecule's coordinate buffer in
// global memory, or the block's window of it staged in shared memory (bead j
// at xw[j - off]).  The arithmetic is the same either way, so are the bits.
struct GlobalX {
  const float4* p;
  __device__ __forceinline__ float4 operator()(int j) const { return p[j]; }
  __device__ __forceinline__ GlobalX from(int b) const { return {p + b}; }
};
struct WindowX {
  const float4* p;  // shared memory
  int off;
  __device__ __forceinline__ float4 operator()(int j) const { return p[j - off]; }
  __device__ __forceinline__ WindowX from(int b) const { return {p, off - b}; }
};

// A lane's share of a chunk of kV = 16 entries of a repulsive pair-list row:
// entries lane + c * G, which pl_at lays into one word (at G = 2 into two).
// As 2-byte loads, each with its bounds test, the indexes took as many loads as
// the coordinates; now the next chunk's word is on its way while one is summed.
// us per 50 steps at 4 lanes, list rebuilds included: 50,000 beads 1,317 -> 1,285,
// half of the ensemble of 512 1,886 -> 1,830 (without the read-ahead 50,000 beads
// in one kernel 1,449 -> 1,431 against 1,475 -> 1,425).
template <int G>
__device__ __forceinline__ uint2 chunk_word(const uint2* chunk, int lane) {
  if (G >= 16) return make_uint2(reinterpret_cast<const unsigned short*>(chunk)[pl_at(lane)], 0u);
  return chunk[lane & 3];  // at G = 8 lanes l and l + 4 share a word
}
template <int G>
__device__ __forceinline__ void chunk_partners(uint2 w, const uint2* chunk, int lane,
                                               unsigned (&jj)[kV / G]) {
  constexpr int kC = kV / G;
  if (G >= 16) {
    jj[0] = w.x;
  } else if (G == 8) {  // entries l, l + 8 of the word's l, l + 4, l + 8, l + 12
    const unsigned half = lane & 4 ? 0x4432u : 0x4410u;
    jj[0] = __byte_perm(w.x, 0u, half);
    jj[1 % kC] = __byte_perm(w.y, 0u, half);
  } else {
    jj[0] = w.x & 0xffffu;
    jj[(4 / G) % kC] = w.x >> 16;
    jj[(8 / G) % kC] = w.y & 0xffffu;
    jj[(12 / G) % kC] = w.y >> 16;
    if (G == 2) {
      const uint2 v = chunk[lane + 2];
      jj[1] = v.x & 0xffffu;
      jj[3 % kC] = v.x >> 16;
      jj[5 % kC] = v.y & 0xffffu;
      jj[7 % kC] = v.y >> 16;
    }
  }
}

// The kV partial sums of a bead, kC = kV / G in each of its G lanes: upper
// levels of the fixed tree inside the lane, lower levels by shuffles; the
// result (and fene_bad of any lane) in every lane.
template <int G>
__device__ __forceinline__ void group_sum(float (&ax)[kV / G], float (&ay)[kV / G], float (&az)[kV / G],
                                          float& fx, float& fy, float& fz, bool& fene_bad) {
  constexpr int kC = kV / G;
  const unsigned gmask = (G == 32) ? 0xffffffffu
                                   : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
#pragma unroll
  for (int off = kV / 2; off >= G; off >>= 1) {
    const int oc = off / G;
#pragma unroll
    for (int c = 0; c < kC; ++c)
      if (c < oc) {
        ax[c] = __fadd_rn(ax[c], ax[c + oc]);
        ay[c] = __fadd_rn(ay[c], ay[c + oc]);
        az[c] = __fadd_rn(az[c], az[c + oc]);
      }
  }
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) {
    ax[0] = __fadd_rn(ax[0], __shfl_xor_sync(gmask, ax[0], off));
    ay[0] = __fadd_rn(ay[0], __shfl_xor_sync(gmask, ay[0], off));
    az[0] = __fadd_rn(az[0], __shfl_xor_sync(gmask, az[0], off));
  }
  fene_bad = __any_sync(gmask, fene_bad);
  fx = ax[0];
  fy = ay[0];
  fz = az[0];
}

// The conservative force on bead i at step n's coordinates, summed by the G lanes of its group over
// its rows (bonds, angles, native pair list, repulsive pair list) into the
// lane's kC virtual-lane accumulators, reduced to lane 0 of the group.
// Forces are summed in a fixed order whatever G is: entry e of a row
// accumulates into virtual lane e % kV (in increasing e), and the kV partial
// sums combine in one fixed binary tree (pairs v, v + kV/2, then v, v + kV/4,
// ...).  Each physical lane holds kC = kV / G virtual lanes and does the
// upper tree levels locally, the rest by shuffles.  So every G gives
// bit-identical forces, and G is free to tune per context.
template <int G, bool UNI, bool wrap_list, class XS>
__device__ __forceinline__ void bead_force_w(const DevSys& s, const XS& X, int i, int m1, long long n,
                                           int lane, int2 br, int2 ar, int abase, int acnt, int rcnt,
                                           float& fx, float& fy, float& fz, bool& fene_bad) {
  constexpr int kC = kV / G;
  float ax[kC], ay[kC], az[kC];
#pragma unroll
  for (int c = 0; c < kC; ++c) ax[c] = ay[c] = az[c] = 0.f;
  const float4 xi = X(i);
  const float boxl = s.boxl;
  const bool wrap = s.grid[m1].wrap != 0;
  const long long rbase = (long long)i * s.nl_stride;
  const uint2* prow = reinterpret_cast<const uint2*>(s.pl_j + rbase);
  uint2 next = make_uint2(0u, 0u);
  if (rcnt > 0) next = chunk_word<G>(prow, lane);

  // Bonded, angle and native terms share one index space [bonds | angles |
  // natives]; a bead has a handful of them, usually one pass.
  const int nba = br.y + ar.y;
  const int nsmall = nba + acnt;
  for (int base = 0; base < nsmall; base += kV) {
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      const int e = base + lane + c * G;
      if (e >= nsmall) break;
      int j;
      float r0 = 0.f, eps = 0.f;
      if (e < br.y) {
        j = s.bond_j[br.x + e];
        r0 = s.bond_r0[br.x + e];
      } else if (e < nba) {
        j = s.ang_j[ar.x + e - br.y];
      } else {
        const float4 q = s.pl_att[abase + e - nba];
        j = __float_as_int(q.x);
        r0 = q.y;
        eps = q.z;
      }
      const float4 xj = X(j);
      float lx, ly, lz;
      float dx = diff_exact(xj.x, xi.x, lx), dy = diff_exact(xj.y, xi.y, ly),
            dz = diff_exact(xj.z, xi.z, lz);
      if (wrap) min_image3(dx, dy, dz, boxl);
      const float cc = small_coeff(s, e < br.y ? 0 : e < nba ? 1 : 2, dx, dy, dz, lx, ly, lz, r0,
                                   eps, fene_bad);
      acc3(ax[c], ay[c], az[c], cc, dx, dy, dz);
    }
  }

  // Non-native repulsion, kC loads in flight per lane per chunk of kV entries
  const RepConst rc = rep_const(s);
  // pair-list partners are stored relative to the molecule's first bead
  const XS Xm = X.from(s.mol[m1].start);
  for (int base = 0; base < rcnt; base += kV, prow += kV / 4) {
    const uint2 w = next;
    if (base + kV < rcnt) next = chunk_word<G>(prow + kV / 4, lane);
    unsigned jj[kC];
    chunk_partners<G>(w, prow, lane, jj);
    float4 xx[kC];
#pragma unroll
    for (int c = 0; c < kC; ++c) xx[c] = Xm(jj[c]);
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      // past the row end xx[c] is bead i itself: d2 = 0 fails the tolerance
      // test and contributes exactly 0, so no branch is needed
      rep_entry<UNI, wrap_list>(rc, xi, xx[c], ax[c], ay[c], az[c]);
    }
  }
  group_sum<G>(ax, ay, az, fx, fy, fz, fene_bad);
}

// Compiled with and without the minimum image of the repulsive pairs (the same
// for a whole molecule).
template <int G, bool UNI, class XS>
__device__ __forceinline__ void bead_force(const DevSys& s, const XS& X, int i, int m1, long long n,
                                           int lane, int2 br, int2 ar, int abase, int acnt, int rcnt,
                                           float& fx, float& fy, float& fz, bool& fene_bad) {
  if (list_image_taken(s, m1, n))
    bead_force_w<G, UNI, true>(s, X, i, m1, n, lane, br, ar, abase, acnt, rcnt, fx, fy, fz, fene_bad);
  else
    bead_force_w<G, UNI, false>(s, X, i, m1, n, lane, br, ar, abase, acnt, rcnt, fx, fy, fz, fene_bad);
}

}  // namespace sop
