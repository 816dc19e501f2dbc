// Host <-> device traffic: the state of molecules packed for the host, states
// and whole molecules unpacked from it.  A buffer here is pinned host memory
// that the kernel reads or writes in place, or device memory that is copied
// whole.
//
// Bound by latency: a call on a small context is as long as its launches,
// copies and waits (18 us for the shortest copy and its wait, a launch and its
// wait half that), and a copy of 12 of every 16 bytes runs row by row (15 us at
// 50,000 beads against 2 us for the packed one).  So one kernel moves all
// arrays of a call, a word a thread: words of packed xyz lie side by side, so
// the accesses across the link are whole lines and only those to device memory
// have holes.
#include <algorithm>

#include "io.cuh"

namespace sop {

constexpr int kIoThreads = 256;

static inline unsigned io_blocks(long long words) {
  return (unsigned)std::max<long long>(1, (words + kIoThreads - 1) / kIoThreads);
}

__global__ void __launch_bounds__(kIoThreads) k_pack_state(DevSys s, int m, int start, int n, StateOut o) {
  const int t = blockIdx.x * kIoThreads + threadIdx.x;
  const long long step = s.mol_step[m];
  if (t == 0 && o.step) {
    *o.step = step;
    *o.status = s.mol_status[m];
  }
  if (t >= 3 * n) return;
  const int cur = (int)(step & 1), b = t / 3, c = t - 3 * b;
  const float4* src[4] = {s.p[cur], s.x[cur], s.v, s.f};
#pragma unroll
  for (int a = 0; a < 4; ++a)
    if (o.a[a]) o.a[a][t] = reinterpret_cast<const float*>(src[a] + start + b)[c];
}

// The new state goes to both coordinate buffers, the bead types (the last
// word of x) stay.
__global__ void __launch_bounds__(kIoThreads) k_unpack_state(DevSys s, int start, int n,
                                                             const float* __restrict__ pos,
                                                             const float* __restrict__ unc,
                                                             const float* __restrict__ vel) {
  const int t = blockIdx.x * kIoThreads + threadIdx.x;
  if (t >= 3 * n) return;
  const int b = t / 3, c = t - 3 * b;
  auto put = [&](float4* dst, float v, bool clear) {
    float* d = reinterpret_cast<float*>(dst + start + b);
    d[c] = v;
    if (clear && c == 0) d[3] = 0.f;
  };
  if (unc) {
    const float v = unc[t];
    put(s.x[0], v, false);
    put(s.x[1], v, false);
  }
  if (pos) {
    const float v = pos[t];
    put(s.p[0], v, true);
    put(s.p[1], v, true);
  }
  if (vel) put(s.v, vel[t], true);
}

// A job per blockIdx.y: its final coordinates and velocities to the host, and
// its slot freed (the molecule inactive, its beads unowned).
__global__ void __launch_bounds__(kIoThreads) k_retire(DevSys s, MolConst* mol, const RetireJob* jobs) {
  const RetireJob j = jobs[blockIdx.y];
  const int t = blockIdx.x * kIoThreads + threadIdx.x;
  if (t < (int)(sizeof(MolConst) / sizeof(int))) reinterpret_cast<int*>(mol + j.e.m)[t] = 0;
  if (t >= 3 * j.e.n) return;
  const int b = t / 3, c = t - 3 * b;
  j.unc[t] = reinterpret_cast<const float*>(s.x[j.cur] + j.e.start + b)[c];
  j.vel[t] = reinterpret_cast<const float*>(s.v + j.e.start + b)[c];
  if (c == 0) s.mol_of[j.e.start + b] = -1;
}

// A molecule per blockIdx.y, from its rows on the host: what upload_staged
// does with a copy or a clear per array.
__global__ void __launch_bounds__(kIoThreads) k_install(DevSys s, MolConst* mol, const InstallJob* jobs) {
  const InstallJob& j = jobs[blockIdx.y];
  const int n = j.n, t0 = blockIdx.x * kIoThreads + threadIdx.x, all = gridDim.x * kIoThreads;
  auto copy = [&](void* dst, const void* src, int words) {
    for (int t = t0; t < words; t += all) static_cast<int*>(dst)[t] = static_cast<const int*>(src)[t];
  };
  for (int t = t0; t < 4 * n; t += all) {
    const float x = j.x0[t], p = j.p0[t];
    reinterpret_cast<float*>(s.x[0] + j.o)[t] = x;
    reinterpret_cast<float*>(s.x[1] + j.o)[t] = x;
    reinterpret_cast<float*>(s.p[0] + j.o)[t] = p;
    reinterpret_cast<float*>(s.p[1] + j.o)[t] = p;
    reinterpret_cast<float*>(s.incr + j.o)[t] = 0.f;
    reinterpret_cast<float*>(s.f + j.o)[t] = 0.f;
  }
  copy(s.v + j.o, j.v0, 4 * n);
  copy(s.bond_row + j.o, j.brow, 2 * n);
  copy(s.ang_row + j.o, j.arow, 2 * n);
  copy(s.nat_row + j.o, j.nrow, 2 * n);
  copy(s.bond_j + j.ob, j.bj, j.nb);
  copy(s.bond_r0 + j.ob, j.br, j.nb);
  copy(s.ang_j + j.oa, j.aj, j.na);
  copy(s.nat_j + j.on, j.nj, j.nn);
  copy(s.nat_par + j.on, j.np, 4 * j.nn);
  copy(s.nat_rc2 + j.on, j.nr, 2 * j.nn);
  for (int t = t0; t < n; t += all) {
    s.nl_cnt[j.o + t] = s.pl_cnt[j.o + t] = 0;
    s.nl_att_cnt[j.o + t] = s.pl_att_cnt[j.o + t] = 0;
    s.mol_of[j.o + t] = j.slot;
  }
  copy(mol + j.slot, &j.mc, (int)(sizeof(MolConst) / sizeof(int)));
  if (t0 == 0) {
    s.mol_step[j.slot] = j.step0;
    s.mol_status[j.slot] = 0;
  }
}

void launch_pack_state(const DevSys& s, int m, int start, int n, const StateOut& o, cudaStream_t st) {
  const bool any = o.a[0] || o.a[1] || o.a[2] || o.a[3];
  k_pack_state<<<any ? io_blocks(3LL * n) : 1, kIoThreads, 0, st>>>(s, m, start, any ? n : 0, o);
}

void launch_unpack_state(const DevSys& s, int start, int n, const float* pos, const float* unc,
                         const float* vel, cudaStream_t st) {
  if (pos || unc || vel)
    k_unpack_state<<<io_blocks(3LL * n), kIoThreads, 0, st>>>(s, start, n, pos, unc, vel);
}

void launch_retire(const DevSys& s, MolConst* mol, const RetireJob* jobs, int count, int most,
                   cudaStream_t st) {
  k_retire<<<dim3(io_blocks(3LL * most), count), kIoThreads, 0, st>>>(s, mol, jobs);
}

void launch_install(const DevSys& s, MolConst* mol, const InstallJob* jobs, int count, int most,
                    cudaStream_t st) {
  k_install<<<dim3(io_blocks(4LL * most), count), kIoThreads, 0, st>>>(s, mol, jobs);
}

}  // namespace sop
