// What the host hands to the kernels of kernels_io.cu and to the energy sums.
#pragma once
#include "sop_dev.cuh"

namespace sop {

// Where a molecule's state goes, packed xyz (null: not asked for): wrapped
// and unwrapped coordinates, velocities, forces; its step and status.
struct StateOut {
  float* a[4];
  long long* step;
  int* status;
};

// A molecule whose energy is summed: its beads, its slot and its first group
// of partial sums.
struct EnergyJob {
  int start, n, m, part;
};

// A served job that leaves its slot.
struct RetireJob {
  EnergyJob e;
  int cur;  // coordinate buffer of its last step
  float *unc, *vel;
};

// A molecule that takes a slot: its pool ranges and its rows.
struct InstallJob {
  int n, nb, na, nn;  // beads; entries of the bond, angle and native rows
  int slot;
  long long o, ob, oa, on, step0;
  MolConst mc;
  const float *x0, *p0, *v0;
  const int2 *brow, *arow, *nrow;
  const int *bj, *aj, *nj;
  const float *br, *np, *nr;
};

void launch_pack_state(const DevSys& s, int m, int start, int n, const StateOut& o, cudaStream_t st);
void launch_unpack_state(const DevSys& s, int start, int n, const float* pos, const float* unc,
                         const float* vel, cudaStream_t st);
void launch_retire(const DevSys& s, MolConst* mol, const RetireJob* jobs, int count, int most,
                   cudaStream_t st);
void launch_install(const DevSys& s, MolConst* mol, const InstallJob* jobs, int count, int most,
                    cudaStream_t st);
// Of one molecule (jobs null) or of `count` of up to e.n beads each, terms to out[4 k ..].
void launch_energy(const DevSys& s, const EnergyJob& e, const RetireJob* jobs, int count,
                   double* part, double* out, double k_bnd_R0sq_half, cudaStream_t st);

}  // namespace sop
