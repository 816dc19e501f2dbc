// Per-bead device code of the step, shared by the step kernels
// (kernels_step.cu, kernels_tile.cu): the terms of the force and the completion
// of a bead (noise, velocity, look-ahead position).  All kernels run the same
// operations in the same order, so every form of the step gives the same bits.
#pragma once
#include "sop_dev.cuh"
#include "../../include/sop_gpu.h"

namespace sop {

constexpr int kV = 16;  // virtual lanes of the fixed force-summation order

// Every rounding of the per-entry arithmetic and of the accumulation is
// written out (one rounding per operation), so the compiler cannot contract
// it differently in different instantiations: the sums are then the same
// bits for every lane-group width.
__device__ __forceinline__ void acc3(float& ax, float& ay, float& az, float c, float dx, float dy,
                                     float dz) {
  ax = __fmaf_rn(c, dx, ax);
  ay = __fmaf_rn(c, dy, ay);
  az = __fmaf_rn(c, dz, az);
}

__device__ __forceinline__ float d2_plain(float dx, float dy, float dz) {
  return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// 1/x by the approximate reciprocal of the PTX ISA: the same bits as
// __fdividef(1, x) for every x that is not denormal (tests/test_gpu_reciprocal.py
// compares them all), in less time: us per 50 steps of the ensemble of 512 3,292 ->
// 3,172, of 50,000 beads 1,372 -> 1,318.  For the repulsive terms alone: a denormal
// d^2, which it takes for zero, fails their tolerance test, so its reciprocal is
// never used.
__device__ __forceinline__ float rcp_normal(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Force coefficient of one bonded / angle / native entry (type 0 / 1 / 2):
// the reference kernels' formulas, with the compensated d^2 - r0^2 wherever
// a difference from the native distance enters.
__device__ __forceinline__ float small_coeff(const DevSys& s, int type, float dx, float dy, float dz,
                                             float lx, float ly, float lz, float r0, float eps,
                                             bool& fene_bad) {
  const float d2 = d2_plain(dx, dy, dz);
  if (type == 0) {
    // FENE: force on i = +k dev / (r (1 - dev^2/R0^2)) * d  (energy.cu:252-271);
    // dev carries the compensated d^2 - r0^2, so approximate reciprocals
    // (a few ulps) keep the term well inside the force tolerance
    const float r = __fmul_rn(d2, rsqrtf(d2));
    const float dev = __fmul_rn(d2_minus_r02(dx, dy, dz, lx, ly, lz, r0),
                                __fdividef(1.0f, __fadd_rn(r, r0)));
    const float w = __fsub_rn(1.0f, __fmul_rn(__fmul_rn(dev, dev), s.inv_R0sq));
    fene_bad |= !(fabsf(dev) < s.R0);
    return __fmul_rn(__fmul_rn(s.k_bnd, dev), __fdividef(1.0f, __fmul_rn(r, w)));
  }
  if (type == 1) {
    // i,i+2 soft sphere: force on i = -6 eps sigma^6 / d^8 * d  (energy.cu:335-360)
    const float inv = __fdividef(1.0f, d2);
    const float inv2 = __fmul_rn(inv, inv);
    return __fmul_rn(-s.f_ss, __fmul_rn(inv2, inv2));
  }
  // native LJ 12-6 (energy.cu:468-507): co1 = -12 eps / d^2 (s^6 - s^3),
  // s = r0^2 / d^2, as -12 eps / d^2 s^3 (s - 1)(s^2 + s + 1) with
  // s - 1 = -(d^2 - r0^2) / d^2; pairs with d^2 <= 1e-7 r0^2 are skipped.
  const float r02 = __fmul_rn(r0, r0);
  const float inv = __fdividef(1.0f, d2);
  const float sr = __fmul_rn(r02, inv);
  const float sm1 = __fmul_rn(-d2_minus_r02(dx, dy, dz, lx, ly, lz, r0), inv);
  const float s3 = __fmul_rn(__fmul_rn(sr, sr), sr);
  const float poly = __fadd_rn(__fadd_rn(__fmul_rn(sr, sr), sr), 1.0f);
  const float c =
      __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(-12.0f, eps), inv), __fmul_rn(s3, sm1)), poly);
  return d2 > __fmul_rn(1.0e-7f, r02) ? c : 0.0f;
}

// One non-native repulsion (energy.cu:536-581): co1 = -6 eps / d^2 (2 (s/r)^12 +
// (s/r)^6) [rep6: -6 eps / d^2 (s/r)^6]; pairs with d^2 <= 1e-7 sigma are
// skipped.  A system of one bead type (UNI) uses its sigma as a constant.
// wrap is false when no listed pair of the molecule can reach boxl/2 (MolGrid):
// the minimum image is the identity.
// (As a run-time test of every entry it cost 18% of the step's instructions
// at 4 lanes per bead.)
struct RepConst {
  float g11, g12, g22, t11, t12, t22, ce, two, q4, boxl;
};
__device__ __forceinline__ RepConst rep_const(const DevSys& s) {
  return {s.sig2[1][1],      s.sig2[1][2],           s.sig2[2][2],   s.rep_tol[1][1],
          s.rep_tol[1][2],   s.rep_tol[2][2],        -6.0f * s.eps_rep,
          s.rep6 ? 0.0f : 2.0f, 0.25f * s.boxl,      s.boxl};
}
template <bool UNI, bool wrap>
__device__ __forceinline__ void rep_entry(const RepConst& rc, float4 xi, float4 xj, float& ax,
                                          float& ay, float& az) {
  float dx = __fsub_rn(xj.x, xi.x), dy = __fsub_rn(xj.y, xi.y), dz = __fsub_rn(xj.z, xi.z);
  // |dx| + |dy| + |dz| bounds every component: one test for the rare wrap
  if (wrap && fabsf(dx) + fabsf(dy) + fabsf(dz) > rc.q4) min_image3(dx, dy, dz, rc.boxl);
  const float d2 = d2_plain(dx, dy, dz);
  float sg2 = rc.g11, tol = rc.t11;
  if (!UNI) {
    const int ti = type_of(xi), tj = type_of(xj);
    sg2 = pick_type_pair(rc.g11, rc.g12, rc.g22, ti, tj);
    tol = pick_type_pair(rc.t11, rc.t12, rc.t22, ti, tj);
  }
  const float inv = rcp_normal(d2);
  const float u = __fmul_rn(sg2, inv);
  const float u3 = __fmul_rn(__fmul_rn(u, u), u);
  const float cc =
      (d2 > tol) ? __fmul_rn(__fmul_rn(__fmul_rn(rc.ce, inv), u3), __fmaf_rn(rc.two, u3, 1.0f)) : 0.0f;
  acc3(ax, ay, az, cc, dx, dy, dz);
}

// Marker bits in the w of a bead's force sum (0: not summed this step).
constexpr int kSummed = 1;
constexpr int kFeneBad = 2;   // a bond at or past R0
constexpr int kOddStep = 4;   // the step is odd: coordinates in buffer 1

// The force sum's w: the marker bits of finish_bead (summed, a bond past R0,
// the parity of the step, which selects the coordinate buffers).
__device__ __forceinline__ float4 marked_sum(float fx, float fy, float fz, bool fene_bad,
                                             long long n) {
  return make_float4(fx, fy, fz,
                     __int_as_float(kSummed | (fene_bad ? kFeneBad : 0) |
                                    ((int)(n & 1) ? kOddStep : 0)));
}

// What completing bead b (of molecule m) at step mol_step + STEP + koff needs
// besides its force sum: its state (coordinates from buffer cur, the step's
// parity) and its noise.  None of it is written by the force kernel of the
// same step.
struct BeadState {
  MolConst mc;
  long long nb;
  float4 vi, inc, xo, pi;
  float3 z;
};

// The standard normals of bead b (of a molecule whose first bead is `start`
// and Philox stream `traj`) at step nb: drawn, or injected.
__device__ __forceinline__ float3 bead_noise(const DevSys& s, int b, int start, long long nb,
                                             unsigned traj) {
  if (s.use_noise) {
    const float4 q = s.noise[b];
    return make_float3(q.x, q.y, q.z);
  }
  return noise3((unsigned)(b - start), nb, traj, s.seed_lo, s.seed_hi);
}

template <bool STEP>
__device__ __forceinline__ void load_bead_state(const DevSys& s, int b, int m, int koff, int cur,
                                                BeadState& t) {
  t.mc = s.mol[m];
  t.nb = s.mol_step[m] + (STEP ? 1 : 0) + koff;
  t.vi = s.v[b];
  t.inc = s.incr[b];
  t.xo = s.x[cur][b];
  t.pi = s.p[cur][b];
  t.z = bead_noise(s, b, t.mc.start, t.nb, t.mc.traj);
}

// Completes bead b from its conservative force sum fs, whose w holds the
// marker bits k_step set: noise, status, velocity and the look-ahead
// position update (sop.cu:421-462, energy.cu:588-604).  Every rounding is
// written out.
template <bool STEP>
__device__ __forceinline__ void complete_bead(const DevSys& s, int b, int m, float4 fs, int cur,
                                              const BeadState& t) {
  const int w = __float_as_int(fs.w);
  const MolConst& mc = t.mc;
  float4 vi = t.vi;
  float4 inc = t.inc;
  const float4 xo = t.xo;
  const float4 pi = t.pi;
  const float3 z = t.z;
  const float fxx = __fmaf_rn(mc.sigma_f, z.x, fs.x);
  const float fyy = __fmaf_rn(mc.sigma_f, z.y, fs.y);
  const float fzz = __fmaf_rn(mc.sigma_f, z.z, fs.z);
  int st = 0;
  if (w & kFeneBad) st |= SOP_MOL_FENE_RANGE;
  if (!(isfinite(fxx) && isfinite(fyy) && isfinite(fzz))) st |= SOP_MOL_NONFINITE;
  if (st) atomicOr(s.mol_status + m, st);
  s.f[b] = make_float4(fxx, fyy, fzz, 0.f);
  // step 0 is the initial force evaluation (sop.cu:180-186): velocities stay
  if (STEP && t.nb > 0 && !mc.t_zero) {
    vi = make_float4(__fmaf_rn(mc.a3, inc.x, __fmul_rn(mc.a4, fxx)),
                     __fmaf_rn(mc.a3, inc.y, __fmul_rn(mc.a4, fyy)),
                     __fmaf_rn(mc.a3, inc.z, __fmul_rn(mc.a4, fzz)), 0.f);
    s.v[b] = vi;
  }
  inc = make_float4(__fmaf_rn(mc.a1, vi.x, __fmul_rn(mc.a2, fxx)),
                    __fmaf_rn(mc.a1, vi.y, __fmul_rn(mc.a2, fyy)),
                    __fmaf_rn(mc.a1, vi.z, __fmul_rn(mc.a2, fzz)), 0.f);
  s.incr[b] = inc;
  s.x[cur ^ 1][b] = make_float4(__fadd_rn(xo.x, inc.x), __fadd_rn(xo.y, inc.y),
                                __fadd_rn(xo.z, inc.z), xo.w);
  const float boxl = s.boxl;
  s.p[cur ^ 1][b] = make_float4(min_image(__fadd_rn(pi.x, inc.x), boxl),
                                min_image(__fadd_rn(pi.y, inc.y), boxl),
                                min_image(__fadd_rn(pi.z, inc.z), boxl), 0.f);
  // moved too far for the minimum image to stay left out until the next look at
  // the molecule's extent (after the stores: ahead of them 0.5% of the small steps)
  const float far = fmaxf(fmaxf(fabsf(inc.x), fabsf(inc.y)), fabsf(inc.z));
  if (!(far <= s.move_least) && !(far <= s.grid[m].move)) {
    if (!s.grid[m].wrap) s.grid[m].wrap = image_mark(t.nb);
    if (!s.grid[m].wrap_list) s.grid[m].wrap_list = image_mark(t.nb);
  }
}

// Completes bead b (of molecule m) from its force sum fs; the step is the
// molecule's mol_step + STEP + koff, as in k_step, and its parity (which
// selects the coordinate buffers) is marked in fs.w.
template <bool STEP>
__device__ __forceinline__ void finish_bead(const DevSys& s, int b, int m, float4 fs, int koff) {
  const int cur = (__float_as_int(fs.w) & kOddStep) ? 1 : 0;
  BeadState t;
  load_bead_state<STEP>(s, b, m, koff, cur, t);
  complete_bead<STEP>(s, b, m, fs, cur, t);
}

}  // namespace sop
