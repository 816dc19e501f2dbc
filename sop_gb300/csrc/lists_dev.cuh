// Device code of the list rebuilds shared by kernels_lists.cu and
// kernels_tile.cu.
#pragma once
#include "sop_dev.cuh"

namespace sop {

// Molecules whose lists a rebuild at block offset koff refreshes: running,
// healthy, and with the step this rebuild precedes (mol_step + koff + 1)
// still within the step budget -- a molecule that has finished keeps the
// lists of its last step, as the reference's loop ends there.
__device__ __forceinline__ bool mol_listed(const DevSys& s, int m, int koff) {
  if (m < 0) return false;
  if (s.only_mol >= 0 && m != s.only_mol) return false;  // its lists and grid stay
  const MolConst& mc = s.mol[m];
  return mc.active && s.mol_status[m] == 0 &&
         !(mc.nsteps >= 0 && s.mol_step[m] + koff >= mc.nsteps);
}

// Coordinates at step mol_step + koff (the positions the rebuild uses).
__device__ __forceinline__ const float4* xbuf(const DevSys& s, int m, int koff) {
  return s.x[(int)((s.mol_step[m] + koff) & 1)];
}

// The lanes of a group of L lanes (L divides 32) within its warp.
template <int L>
__device__ __forceinline__ unsigned group_mask(int wl) {
  return L == 32 ? 0xffffffffu : (((1u << L) - 1u) << (wl & ~(L - 1)));
}

// The pair-list rows of bead i of molecule m, rebuilt from the coordinates X by
// the L lanes of a group together: the in-order compaction of the bead's
// neighbour-list row by the pair-list cut-off (sop.cu:835-920 semantics, host
// arithmetic of sop.cu:1737-1810).  Each lane takes 4 consecutive entries per
// round (one 8-byte load, four independent gathers) and a scan across the
// group places the survivors; the attractive pair list is the same over the
// bead's attractive neighbour list.  The lists do not depend on L.
// rep(position, partner within the molecule) and att(position, entry) also get
// every entry of the two rows; nrep / natt are their lengths, in every lane.
//
// Bound by instructions: a round's tests of the row's end are one mask, its
// indexes count from the molecule's first bead on (a test and a select per entry
// before): with a list before every step 50 steps of 1,531 beads 525 -> 504 us,
// of 10,870 beads in 37 molecules 1,010 -> 990 (both against 515 and 1,017 at
// the layout before pl_at).
//
// What the rebuild reads before any coordinate: the row lengths and the
// first round of each row (of the attractive one when kAhead).  Only
// neighbour-list rebuilds write it, so a kernel that follows others which use
// the lists may read it ahead of its wait.
struct PairHead {
  int cnt, acnt, mstart;
  int2 row;     // the bead's native row
  bool wrap, wrap_list;  // the minimum image is taken (MolGrid)
  uint2 j;      // four entries of the repulsive row
  int natj;     // one of the attractive row: partner, squared cut-off, parameters
  float rc2;
  float4 par;
};
template <int L, bool kAhead>
__device__ __forceinline__ PairHead pair_head(const DevSys& s, int i, int m) {
  const int lane = threadIdx.x & (L - 1);
  PairHead h;
  h.cnt = s.nl_cnt[i];
  h.acnt = s.nl_att_cnt[i];
  h.row = s.nat_row[i];
  h.mstart = s.mol[m].start;
  // steps write these too: not ahead of a wait, where whoever calls sets them
  h.wrap = !kAhead && s.grid[m].wrap != 0;
  h.wrap_list = !kAhead && s.grid[m].wrap_list != 0;
  h.j = make_uint2(0, 0);
  if (4 * lane < h.cnt) h.j = reinterpret_cast<const uint2*>(s.nl_j + (long long)i * s.nl_stride)[lane];
  h.natj = 0;
  h.rc2 = 0.f;
  h.par = make_float4(0.f, 0.f, 0.f, 0.f);
  if (kAhead && lane < h.acnt) {
    const int idx = s.nl_att_e[h.row.x + lane];
    h.natj = s.nat_j[idx];
    h.rc2 = s.nat_rc2[idx].y;
    h.par = s.nat_par[idx];
  }
  return h;
}
template <bool UNI, int L, bool kAhead, bool wrap_list, class Rep, class Att>
__device__ __forceinline__ void pair_rows_w(const DevSys& s, const float4* X, int i, const PairHead& h,
                                          Rep rep, Att att, int& nrep, int& natt) {
  const int wl = threadIdx.x & 31;
  const int lane = wl & (L - 1);
  const unsigned gmask = group_mask<L>(wl);
  const float4 xi = X[i];
  const int ti = type_of(xi);
  const float boxl = s.boxl;
  const float r11 = s.rc2_pl_rep[1][1], r12 = s.rc2_pl_rep[1][2], r22 = s.rc2_pl_rep[2][2];
  const unsigned below = (1u << wl) - 1u;  // lanes of the warp before this one
  const long long a = (long long)i * s.nl_stride;
  // rows hold partners relative to the molecule's first bead, 4 per 8 bytes,
  // the last four filled up with some bead of the molecule (k_nl)
  const uint2* row4 = reinterpret_cast<const uint2*>(s.nl_j + a);
  unsigned short* out = s.pl_j + a;
  const float4* Xm = X + h.mstart;
  const unsigned irel = (unsigned)(i - h.mstart);
  const int cnt = h.cnt, acnt = h.acnt;
  const int2 row = h.row;
  int k = 0;
  // each round works on entries loaded the round before (rows are read ahead)
  uint2 jn = 4 * lane < cnt ? h.j : make_uint2(0u, 0u);
  for (int e0 = 0; e0 < cnt; e0 += 4 * L) {
    const int e = e0 + 4 * lane;
    const uint2 jv = jn;
    jn = make_uint2(0u, 0u);
    if (e + 4 * L < cnt) jn = row4[(e0 >> 2) + L + lane];
    const unsigned jq[4] = {jv.x & 0xffffu, jv.x >> 16, jv.y & 0xffffu, jv.y >> 16};
    unsigned pb = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 xj = Xm[jq[q]];
      float dx = __fsub_rn(xj.x, xi.x), dy = __fsub_rn(xj.y, xi.y),
            dz = __fsub_rn(xj.z, xi.z);
      if (wrap_list) min_image3(dx, dy, dz, boxl);
      const bool p = d2_exact(dx, dy, dz) < (UNI ? r11 : pick_type_pair(r11, r12, r22, ti, type_of(xj)));
      pb |= (p ? 1u : 0u) << q;
    }
    const int left = cnt - e;  // the lane's entries of the row
    if (left < 4) pb &= left > 0 ? (1u << left) - 1u : 0u;
    const int c = __popc(pb);
    int incl = c;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
      const int t = __shfl_up_sync(gmask, incl, o, L);
      if (lane >= o) incl += t;
    }
    int pos = k + incl - c;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (pb & (1u << q)) {
        rep(pos, (int)jq[q]);
        out[pl_at(pos++)] = (unsigned short)jq[q];
      }
    k += __shfl_sync(gmask, incl, L - 1, L);
  }
  // the last chunk filled up with the bead itself
  if (k + lane < ((k + 15) & ~15)) out[pl_at(k + lane)] = (unsigned short)irel;
  if (L < 16 && k + lane + L < ((k + 15) & ~15)) out[pl_at(k + lane + L)] = (unsigned short)irel;
  if (lane == 0) s.pl_cnt[i] = k;
  int ka = 0;
  for (int e0 = 0; e0 < acnt; e0 += L) {
    const int e = e0 + lane;
    bool pass = false;
    int j = 0;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (e < acnt) {
      j = h.natj;
      float rc2 = h.rc2;
      q = h.par;
      if (!kAhead || e0 > 0) {
        const int idx = s.nl_att_e[row.x + e];
        // the contact's partner, cut-off and parameters in one round of loads
        j = s.nat_j[idx];
        rc2 = s.nat_rc2[idx].y;
        q = s.nat_par[idx];
      }
      const float4 xj = X[j];
      float dx = __fsub_rn(xj.x, xi.x), dy = __fsub_rn(xj.y, xi.y),
            dz = __fsub_rn(xj.z, xi.z);
      if (h.wrap) min_image3(dx, dy, dz, boxl);
      pass = d2_exact(dx, dy, dz) < rc2;
    }
    const unsigned mask = __ballot_sync(gmask, pass) & gmask;
    if (pass) {
      const int pos = ka + __popc(mask & below);
      const float4 entry = make_float4(__int_as_float(j), q.x, q.y, q.z);
      att(pos, entry);
      s.pl_att[row.x + pos] = entry;
    }
    ka += __popc(mask);
  }
  if (lane == 0) s.pl_att_cnt[i] = ka;
  nrep = k;
  natt = ka;
}

// Compiled with and without the minimum image of the repulsive pairs (the same
// for a whole molecule).
template <bool UNI, int L, bool kAhead, class Rep, class Att>
__device__ __forceinline__ void pair_rows(const DevSys& s, const float4* X, int i, const PairHead& h,
                                          Rep rep, Att att, int& nrep, int& natt) {
  if (h.wrap_list) pair_rows_w<UNI, L, kAhead, true>(s, X, i, h, rep, att, nrep, natt);
  else pair_rows_w<UNI, L, kAhead, false>(s, X, i, h, rep, att, nrep, natt);
}

}  // namespace sop
