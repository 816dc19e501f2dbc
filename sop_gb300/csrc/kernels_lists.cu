// Neighbour-list and pair-list rebuilds (replace update_neighbor_list /
// update_pair_list, sop.cu:704-920, 928-1262, 1456-1706, and the CUDPP radix
// sort + scan they use).
//
// Neighbour list (every nnlup steps):
//   1. binning: each molecule's bounding box, its cell grid (cell edge rc/S,
//      S=1..3 chosen so a cell holds ~4 beads; S=1..4 and ~1 bead from 10,000
//      beads up; molecules whose extent + rc reaches boxl, where the minimum
//      image matters, fall back to index-chunked cells that scan all pairs), a
//      counting sort of its beads into cells, cells sorted by bead id so every
//      later order is deterministic, coordinates staged in that order.  A
//      molecule's cells start at cell_base and its staged beads at its first
//      bead, so molecules are binned independently: one block per molecule,
//      in shared memory (k_bin_mol); molecules past kBinMolBeads by a chain of
//      kernels over all their beads (k_bbox, k_grid, k_assign, scan,
//      k_scatter, k_cellsort, k_stage_xs)
//   2. 8 lanes (or a warp) per bead in cell order: the bead against the beads
//      of the cell rows within S along each axis, culled to its own cut-off
//      sphere; predicate = the reference's FP32 host filter (d^2 < rcut^2,
//      |i-j| > 2, not native); one pass writes fixed-stride rows (overflow:
//      regrow).  The attractive neighbour list filters the bead's native row.
//                                                                          k_nl
// Pair list (every nplup steps): eight lanes per bead, beads in chain order,
// compact its neighbour-list row in row order (k_pl).
#include "lists_dev.cuh"

namespace sop {

// ------------------------------------------------------------------ scan
// Exclusive scan of n ints: out[0..n], out[n] = total.  Three kernels:
// per-block reduce, one-block scan of the block sums, per-block apply.
constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int warp_incl_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and the block total in *total.  The total has its own slot: with
// 1,024 threads all 32 warp slots hold prefixes.
__device__ __forceinline__ int block_excl_scan(int v, int* total) {
  __shared__ int warp_sums[32];
  __shared__ int block_total;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = warp_incl_scan(v);
  if (lane == 31) warp_sums[w] = incl;
  __syncthreads();
  if (w == 0) {
    int nw = (blockDim.x + 31) >> 5;
    int s = lane < nw ? warp_sums[lane] : 0;
    int si = warp_incl_scan(s);
    if (lane < nw) warp_sums[lane] = si - s;
    if (lane == 31) block_total = si;
  }
  __syncthreads();
  int res = incl - v + warp_sums[w];
  *total = block_total;
  __syncthreads();
  return res;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const int* __restrict__ in, long long n,
                                                               int* __restrict__ block_sums) {
  long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) s += in[base + k];
  int total;
  block_excl_scan(s, &total);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_top(int* __restrict__ block_sums, int nblocks) {
  int carry = 0;
  for (int b0 = 0; b0 < nblocks; b0 += blockDim.x) {
    int b = b0 + threadIdx.x;
    int v = b < nblocks ? block_sums[b] : 0;
    int total;
    int ex = block_excl_scan(v, &total);
    if (b < nblocks) block_sums[b] = ex + carry;
    carry += total;
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const int* __restrict__ in, long long n,
                                                              const int* __restrict__ block_sums,
                                                              int* __restrict__ out) {
  long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  int total;
  int ex = block_excl_scan(s, &total) + block_sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = ex;
    ex += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = ex;
}

// ---------------------------------------------------------------- grids
// First cell of the molecule whose beads start at `start`.  A molecule of n
// beads has at most 2 n cells (n / 32 chunks when every pair is scanned) and
// one more entry of cell_start, which 3 n hold, so the ranges of molecules are
// apart wherever their beads are.
__device__ __forceinline__ int cell_base(int start) { return 3 * start; }

__device__ __forceinline__ bool bins_by_chain(const DevSys& s, int m, int koff) {
  return mol_listed(s, m, koff) && s.mol[m].n > kBinMolBeads;
}

__global__ void k_bbox_reset(DevSys s) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= s.nmol) return;
  unsigned* b = s.bbox + 7 * m;
  b[0] = b[1] = b[2] = f2ord(INFINITY);
  b[3] = b[4] = b[5] = f2ord(-INFINITY);
  b[6] = f2ord(0.0f);
}

// The furthest a coordinate of bead i moved in its last look-ahead.
__device__ __forceinline__ float last_move(const DevSys& s, int i) {
  const float4 d = s.incr[i];
  return fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
}

__global__ void k_bbox(DevSys s, int koff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int m = (i < s.nlive) ? s.mol_of[i] : -1;
  bool ok = bins_by_chain(s, m, koff);
  unsigned act = __ballot_sync(0xffffffffu, ok);
  if (!ok) return;
  float4 x = xbuf(s, m, koff)[i];
  unsigned peers = __match_any_sync(act, m);
  const unsigned moved = __reduce_max_sync(peers, f2ord(last_move(s, i)));
  unsigned lo[3] = {f2ord(x.x), f2ord(x.y), f2ord(x.z)};
  unsigned mn[3], mx[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = __reduce_min_sync(peers, lo[a]);
    mx[a] = __reduce_max_sync(peers, lo[a]);
  }
  if ((threadIdx.x & 31) == __ffs(peers) - 1) {
    unsigned* b = s.bbox + 7 * m;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      atomicMin(b + a, mn[a]);
      atomicMax(b + 3 + a, mx[a]);
    }
    atomicMax(b + 6, moved);
  }
}

// The cell grid of a molecule of n beads within the bounds b (ordered floats:
// three lower, three upper, the furthest last move); old: its grid so far.
__device__ __forceinline__ MolGrid make_grid(const DevSys& s, int n, const unsigned* b, int base,
                                             const MolGrid& old) {
  MolGrid g = {};
  float lo[3], ext[3];
  for (int a = 0; a < 3; ++a) {
    lo[a] = ord2f(b[a]);
    ext[a] = ord2f(b[3 + a]) - lo[a];
  }
  const float rc = s.rc_nl_rep_max;
  bool periodic = false;
  for (int a = 0; a < 3; ++a) periodic |= !(ext[a] + rc < s.boxl);  // also true for NaN extents
  // Separations inside the box [lo, lo + ext] never exceed ext (rounding is
  // monotone), and below boxl/2 the minimum image leaves them unchanged
  // (rint(d / boxl) is 0).  The steps and pair-list filters until the next
  // rebuild use the same flag, so the room to boxl/2, a cut-off at least, is
  // shared out over them as g.move.
  bool wrap = !(s.move_share > 0.0f);  // never rebuilt: always
  for (int a = 0; a < 3; ++a) wrap |= !(ext[a] + rc < 0.5f * s.boxl);
  if (periodic || n <= 96) {
    g.brute = 1;
  } else {
    float vol = fmaxf((ext[0] + 1.0f) * (ext[1] + 1.0f) * (ext[2] + 1.0f), 1.0f);
    float rho = (float)n / vol;
    // about 4 beads per cell (S <= 3); a molecule of 10,000 beads or more
    // scans enough cells per bead that finer ones (about 1 bead, S <= 4) cull
    // more candidates than they add rows
    const bool big = n >= 10000;
    const int smax = big ? 4 : 3;
    int S = (int)floorf(rc * cbrtf(rho * (big ? 1.0f : 0.25f)));
    S = S < 1 ? 1 : (S > smax ? smax : S);
    float cs = rc * 1.0001f / (float)S + 1.0e-4f;
    const long long cap = 2LL * n;
    long long tot = 0;
    for (int iter = 0; iter < 64; ++iter) {
      tot = 1;
      for (int a = 0; a < 3; ++a) {
        g.dims[a] = (int)floorf(ext[a] / cs) + 1;
        tot *= g.dims[a];
      }
      if (tot <= cap) break;
      cs *= cbrtf((float)tot / (float)cap) * 1.01f;
      S = (int)ceilf(rc * 1.0001f / cs);
      if (S < 1) S = 1;
    }
    g.S = S;
    g.cs = cs;
    for (int a = 0; a < 3; ++a) g.lo[a] = lo[a];
    g.brute = tot > cap;  // a bound on the cells, not reached: each round takes 1% off at least
  }
  if (g.brute) {
    // every pair is scanned; cells are chunks of 32 consecutive beads
    g.dims[0] = (n + 31) / 32; g.dims[1] = 1; g.dims[2] = 1;
    g.S = g.dims[0];
    g.cs = 0.0f;
    g.lo[0] = g.lo[1] = g.lo[2] = 0.0f;
  }
  // A molecule that cannot come within a cut-off of its own image is binned by
  // plain separations, and lists pairs within a cut-off of each other only:
  // their separations stay below boxl/2 however far the molecule reaches (a
  // 50,000-bead globule, 340 A across, in a box of 500 A).
  const bool wrap_list = wrap && (g.brute || !(s.move_share > 0.0f) || !(4.1f * rc < s.boxl));
  g.wrap = wrap ? kImageTaken : 0;
  g.wrap_list = wrap_list ? kImageTaken : 0;
  g.move = wrap_list ? INFINITY
                     : s.move_share * (0.5f * s.boxl - (wrap ? rc : fmaxf(ext[0], fmaxf(ext[1], ext[2]))));
  // the step that follows reads coordinates one look-ahead past these
  if (!(ord2f(b[6]) <= g.move)) g.wrap = g.wrap_list = kImageTaken;
  if (s.keep_wrap) {  // its pair list stays, and may hold pairs through the image
    if (old.wrap) g.wrap = kImageTaken;
    if (old.wrap_list) g.wrap_list = kImageTaken;
  }
  g.ncell = g.dims[0] * g.dims[1] * g.dims[2];
  g.base = base;
  return g;
}

__device__ __forceinline__ int cell_coord(float v, float lo, float cs, int dim) {
  int c = (int)floorf((v - lo) / cs);
  return c < 0 ? 0 : (c >= dim ? dim - 1 : c);
}

// The cell of a bead (r within its molecule) at x, within its molecule's grid.
__device__ __forceinline__ int cell_of(const MolGrid& g, int r, float4 x) {
  if (g.brute) return r / 32;
  const int cx = cell_coord(x.x, g.lo[0], g.cs, g.dims[0]);
  const int cy = cell_coord(x.y, g.lo[1], g.cs, g.dims[1]);
  const int cz = cell_coord(x.z, g.lo[2], g.cs, g.dims[2]);
  return (cz * g.dims[1] + cy) * g.dims[0] + cx;
}

// Insertion sort of a cell's beads by id (fixes every downstream order).
// Cells hold a handful of beads, so one thread's sort is short.
__device__ __forceinline__ void sort_cell(int* b, int cnt) {
  for (int a = 1; a < cnt; ++a) {
    int v = b[a], k = a;
    while (k > 0 && b[k - 1] > v) { b[k] = b[k - 1]; --k; }
    b[k] = v;
  }
}

// ------------------------------------------------- one block per molecule
// Blocks walk the molecule slots (a served context has many free ones: each
// thread looks at one slot, the block then bins the live ones in turn).  The
// cell counts, their scan and the sorted order stay in shared memory; a
// chain of 11 launches with its counts in L2, or one block for the whole
// context, took 145-158 us for 1,500-13,000 beads and 69 us for 4,000.
__global__ void __launch_bounds__(1024) k_bin_mol(DevSys s, int koff, int most) {
  extern __shared__ int bin_smem[];
  int* first = bin_smem;                                // cells: counts, then first position
  int* order = bin_smem + 2 * most + 1;        // beads in cell order
  __shared__ unsigned bounds[7];
  __shared__ MolGrid grid;
  __shared__ int found[1024];
  __shared__ int nfound;
  const int T = blockDim.x, t = threadIdx.x, lane = t & 31;
  for (long long m0 = blockIdx.x; m0 < s.nmol; m0 += (long long)gridDim.x * T) {
    if (t == 0) nfound = 0;
    __syncthreads();
    const long long mt = m0 + (long long)t * gridDim.x;
    if (mt < s.nmol && mol_listed(s, (int)mt, koff) && s.mol[mt].n <= kBinMolBeads)
      found[atomicAdd(&nfound, 1)] = (int)mt;
    __syncthreads();
    for (int f = 0; f < nfound; ++f) {
      const int m = found[f];
      const int n = s.mol[m].n, start = s.mol[m].start;
      const float4* X = xbuf(s, m, koff) + start;
      if (t < 7) bounds[t] = f2ord(t < 3 ? INFINITY : t < 6 ? -INFINITY : 0.0f);
      __syncthreads();
      unsigned mn[3], mx[3];
      float far = 0.0f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        mn[a] = f2ord(INFINITY);
        mx[a] = f2ord(-INFINITY);
      }
      for (int r = t; r < n; r += T) {
        const float4 x = X[r];
        const unsigned o[3] = {f2ord(x.x), f2ord(x.y), f2ord(x.z)};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          mn[a] = min(mn[a], o[a]);
          mx[a] = max(mx[a], o[a]);
        }
        far = fmaxf(far, last_move(s, start + r));
      }
      const unsigned moved = __reduce_max_sync(0xffffffffu, f2ord(far));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        mn[a] = __reduce_min_sync(0xffffffffu, mn[a]);
        mx[a] = __reduce_max_sync(0xffffffffu, mx[a]);
      }
      if (lane == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          atomicMin(bounds + a, mn[a]);
          atomicMax(bounds + 3 + a, mx[a]);
        }
        atomicMax(bounds + 6, moved);
      }
      __syncthreads();
      if (t == 0) {
        grid = make_grid(s, n, bounds, cell_base(start), s.grid[m]);
        s.grid[m] = grid;
      }
      __syncthreads();
      const int ncell = grid.ncell;
      for (int c = t; c < ncell; c += T) first[c] = 0;
      __syncthreads();
      for (int r = t; r < n; r += T) {
        const int c = cell_of(grid, r, X[r]);
        s.bead_cell[start + r] = grid.base + c;
        s.bead_slot[start + r] = atomicAdd(first + c, 1);
      }
      __syncthreads();
      // exclusive scan: a run of cells per thread
      const int per = (ncell + T - 1) / T, c0 = min(t * per, ncell), c1 = min(c0 + per, ncell);
      int sum = 0;
      for (int c = c0; c < c1; ++c) sum += first[c];
      int total;
      int at = block_excl_scan(sum, &total);
      for (int c = c0; c < c1; ++c) {
        const int v = first[c];
        first[c] = at;
        at += v;
      }
      if (t == 0) first[ncell] = n;
      __syncthreads();
      for (int r = t; r < n; r += T)
        order[first[s.bead_cell[start + r] - grid.base] + s.bead_slot[start + r]] = r;
      __syncthreads();
      for (int c = t; c <= ncell; c += T) {
        if (c < ncell) sort_cell(order + first[c], first[c + 1] - first[c]);
        s.cell_start[grid.base + c] = start + first[c];
      }
      __syncthreads();
      for (int k = t; k < n; k += T) {
        const int r = order[k];
        float4 x = X[r];
        x.w = __int_as_float(((start + r) << 2) | type_of(x));
        s.xs[start + k] = x;
      }
      __syncthreads();  // the next molecule reuses the shared memory
    }
    __syncthreads();
  }
}

// ------------------------------------- the chain, for molecules past that
// Cell counts in cell_cnt, their exclusive scan over all cells in cell_scan;
// a molecule's beads then lie in the order of its cells at
// cell_scan - cell_scan[its first cell] past its first bead.
__global__ void k_grid(DevSys s, int koff) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= s.nmol || !bins_by_chain(s, m, koff)) return;
  unsigned b[7];
  for (int a = 0; a < 7; ++a) b[a] = s.bbox[7 * m + a];
  s.grid[m] = make_grid(s, s.mol[m].n, b, cell_base(s.mol[m].start), s.grid[m]);
}

__global__ void k_assign(DevSys s, int koff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.nlive) return;
  const int m = s.mol_of[i];
  if (!bins_by_chain(s, m, koff)) return;
  const MolGrid g = s.grid[m];
  const int c = g.base + cell_of(g, i - s.mol[m].start, xbuf(s, m, koff)[i]);
  s.bead_cell[i] = c;
  s.bead_slot[i] = atomicAdd(s.cell_cnt + c, 1);
}

__global__ void k_scatter(DevSys s, int koff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.nlive || !bins_by_chain(s, s.mol_of[i], koff)) return;
  s.sorted[s.cell_scan[s.bead_cell[i]] + s.bead_slot[i]] = i;
}

__global__ void k_cellsort(DevSys s) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= s.cell_cap) return;
  const int cnt = s.cell_cnt[c];
  if (cnt > 1) sort_cell(s.sorted + s.cell_scan[c], cnt);
}

// Coordinates staged in cell order, w = (id << 2) | type: a thread per
// position, so the gathers are independent.
__global__ void k_stage_xs(DevSys s, int koff) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= s.cell_scan[s.cell_cap]) return;  // beads that were binned
  const int i = s.sorted[k];
  const int m = s.mol_of[i];
  float4 x = xbuf(s, m, koff)[i];
  x.w = __int_as_float((i << 2) | type_of(x));
  s.xs[s.mol[m].start + k - s.cell_scan[s.grid[m].base]] = x;
}

// Contexts of up to this many bead slots rebuild their lists with a warp
// per bead: at 8 lanes per bead they fill less than a wave of the GPU.
constexpr int kWideListBeads = 16384;

constexpr int kNatRegs = 16;  // native partners held in registers (the rest are read)

// Distance from v to the slab [a, a + w] (0 inside).
// cell_coord with a multiply by the inverse edge: for bounds that carry a
// margin far above its rounding (about 1e-5 cells)
__device__ __forceinline__ int cell_coord_fast(float v, float lo, float inv_cs, int dim) {
  int c = (int)floorf((v - lo) * inv_cs);
  return c < 0 ? 0 : (c >= dim ? dim - 1 : c);
}

__device__ __forceinline__ float slab_dist(float v, float a, float w) {
  return fmaxf(fmaxf(a - v, v - (a + w)), 0.0f);
}

// Attractive neighbour lists, a thread per bead: the bead's native row by its
// own cut-offs, in row order (sop.cu:704-759 semantics), four entries' loads
// in flight.  Within k_nl at 8 lanes per bead the same filter cost 19 us at
// 50,000 beads (registers and idle lanes), as a kernel of its own 6.
__global__ void __launch_bounds__(128) k_att(DevSys s, int koff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.nlive) return;
  const int m = s.mol_of[i];
  if (!mol_listed(s, m, koff)) return;
  if (*s.flags & FLAG_NL_OVERFLOW) return;
  const float4* X = xbuf(s, m, koff);
  const float4 xi = X[i];
  const int2 row = s.nat_row[i];
  constexpr int kB = 4;
  int k = 0;
  for (int e0 = 0; e0 < row.y; e0 += kB) {
    float4 xx[kB];
    float rc2[kB];
#pragma unroll
    for (int c = 0; c < kB; ++c) {
      const int idx = row.x + min(e0 + c, row.y - 1);
      xx[c] = X[s.nat_j[idx]];
      rc2[c] = s.nat_rc2[idx].x;
    }
#pragma unroll
    for (int c = 0; c < kB; ++c) {
      float dx = __fsub_rn(xx[c].x, xi.x), dy = __fsub_rn(xx[c].y, xi.y),
            dz = __fsub_rn(xx[c].z, xi.z);
      min_image3(dx, dy, dz, s.boxl);
      if (e0 + c < row.y && d2_exact(dx, dy, dz) < rc2[c]) s.nl_att_e[row.x + k++] = row.x + e0 + c;
    }
  }
  s.nl_att_cnt[i] = k;
}

// L lanes per bead (8, or a warp for small contexts; the rows do not depend
// on L), beads in cell order (xs), so neighbouring groups share cells and
// candidates.  Each bead scans the cell rows (runs along x) of its grid
// neighbourhood, culled against its own position: rows whose y,z slab lies
// beyond the cut-off are skipped and each row's x range is clipped to the
// chord.  Partners that pass the reference's predicate (sop.cu:768-826 with the
// host arithmetic of sop.cu:1414-1435: d^2 < (fac*sigma or abs)^2 in FP32,
// |i - j| > 2, not a native contact) are written to the bead's fixed-stride row
// in candidate order (group ballot).  The culling is conservative (a 1e-3 A
// margin); membership is decided by the exact predicate alone.  The bead's
// native partners sit in registers.
//
// A warp per bead (L = 32): every lane takes one cell row's bounds, and the rows'
// candidates then form one list that the lanes walk 32 at a time (the row of
// a candidate found by a search over the rows' prefix sums): one row after
// another, the two dependent reads of a row's cells and three idle lanes in
// four made the list of 4,000 beads 25.6 us (20.5 this way, the attractive
// list included).  At 8 lanes per bead the rows fill the lanes and the search
// costs more than it saves (50,000 beads: 304 us against 264), so each row is
// walked by itself.
constexpr int kNlThreads = 256;
template <bool UNI, int L>
__global__ void __launch_bounds__(kNlThreads, 4) k_nl(DevSys s, int koff) {
  const int k = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) / L);
  const int lane = threadIdx.x % L;
  const unsigned wl = threadIdx.x & 31;
  const unsigned gmask = group_mask<L>((int)wl);
  const unsigned below = (1u << wl) - 1u;
  if (k >= s.nlive) return;
  const int m = s.mol_of[k];  // a molecule's staged beads lie in its own bead range
  const float4 xi = s.xs[k];  // (stale unless the molecule was binned)
  const bool frozen = *s.flags & FLAG_NL_OVERFLOW;
  if (!mol_listed(s, m, koff) || frozen) return;
  const int wi = __float_as_int(xi.w);
  const int i = wi >> 2, ti = wi & 3;
  const int mstart = s.mol[m].start;
  const MolGrid g = s.grid[m];
  const bool chain = s.mol[m].n > kBinMolBeads;
  const int* __restrict__ cells = chain ? s.cell_scan : s.cell_start;
  const int shift = chain ? mstart - s.cell_scan[g.base] : 0;
  const int lc = s.bead_cell[i] - g.base;
  const int nx = g.dims[0], ny = g.dims[1], nz = g.dims[2];
  const int cx = lc % nx, cy = (lc / nx) % ny, cz = lc / (nx * ny);
  const int z0 = max(cz - g.S, 0), z1 = min(cz + g.S, nz - 1);
  const int y0 = max(cy - g.S, 0), y1 = min(cy + g.S, ny - 1);
  const int x0 = max(cx - g.S, 0), x1 = min(cx + g.S, nx - 1);
  const float boxl = s.boxl;
  const bool wrap = g.wrap_list != 0;
  const float inv_cs = g.brute ? 0.0f : 1.0f / g.cs;
  const float r11 = s.rc2_nl_rep[1][1], r12 = s.rc2_nl_rep[1][2], r22 = s.rc2_nl_rep[2][2];
  const float rcm = s.rc_nl_rep_max * 1.0001f + 1.0e-3f;
  const float rcm2 = rcm * rcm;
  const int2 nrow = s.nat_row[i];

  if (L == 32) {
    // attractive neighbour list: the bead's native row by its own cut-offs, in
    // row order (sop.cu:704-759 semantics); k_att has it for L = 8
    const float4* X = xbuf(s, m, koff);
    int katt = 0;
    for (int e0 = 0; e0 < nrow.y; e0 += L) {
      const int e = e0 + lane;
      bool pass = false;
      if (e < nrow.y) {
        const float4 xj = X[s.nat_j[nrow.x + e]];
        float dx = __fsub_rn(xj.x, xi.x), dy = __fsub_rn(xj.y, xi.y), dz = __fsub_rn(xj.z, xi.z);
        min_image3(dx, dy, dz, boxl);
        pass = d2_exact(dx, dy, dz) < s.nat_rc2[nrow.x + e].x;
      }
      const unsigned msk = __ballot_sync(gmask, pass);
      if (pass) s.nl_att_e[nrow.x + katt + __popc(msk & below)] = nrow.x + e;
      katt += __popc(msk);
    }
    if (lane == 0) s.nl_att_cnt[i] = katt;
  }
  int nat[kNatRegs];
#pragma unroll
  for (int q = 0; q < kNatRegs; ++q) nat[q] = q < nrow.y ? s.nat_j[nrow.x + q] : -1;
  const long long stride = s.nl_stride;
  unsigned short* row = s.nl_j + (long long)i * stride;  // partners relative to the molecule start
  int cnt = 0;
  // tests candidate xs[jj] and appends it to the row
  auto candidate = [&](int jj, bool valid) {
    bool pass = false;
    int j = 0;
    if (valid) {
      const float4 xj = s.xs[jj];
      const int wj = __float_as_int(xj.w);
      j = wj >> 2;
      if (abs(j - i) > 2) {
        float dx = __fsub_rn(xj.x, xi.x), dy = __fsub_rn(xj.y, xi.y), dz = __fsub_rn(xj.z, xi.z);
        if (wrap) min_image3(dx, dy, dz, boxl);
        pass = d2_exact(dx, dy, dz) < (UNI ? r11 : pick_type_pair(r11, r12, r22, ti, wj & 3));
        if (pass) {
          bool native = false;
#pragma unroll
          for (int q = 0; q < kNatRegs; ++q) native |= (nat[q] == j);
          for (int q = kNatRegs; q < nrow.y && !native; ++q) native = (s.nat_j[nrow.x + q] == j);
          pass = !native;
        }
      }
    }
    const unsigned msk = __ballot_sync(gmask, pass);
    if (pass) {
      const int pos = cnt + __popc(msk & below);
      if (pos < stride) row[pos] = (unsigned short)(j - mstart);
    }
    cnt += __popc(msk);
  };
  // the candidates of cell row (z, y) at squared distance rcm2 - rem: xs[ja .. jb)
  auto row_range = [&](int z, int y, float rem, int& ja, int& jb) {
    int xa = x0, xb = x1;
    if (!g.brute) {
      // the chord only bounds the candidates (the exact predicate decides):
      // an approximate root and reciprocal, widened by 1e-3 A, keep it a
      // superset at a fraction of the cost of the exact operations
      const float w = __fmul_rn(rem, rsqrtf(fmaxf(rem, 1.0e-30f))) * 1.0001f + 1.0e-3f;
      xa = max(x0, cell_coord_fast(xi.x - w, g.lo[0], inv_cs, nx));
      xb = min(x1, cell_coord_fast(xi.x + w, g.lo[0], inv_cs, nx));
    }
    const int rowc = g.base + (z * ny + y) * nx;
    ja = cells[rowc + xa] + shift;
    jb = cells[rowc + xb + 1] + shift;
  };
  if (L < 32) {
    for (int z = z0; z <= z1; ++z) {
      const float dz = g.brute ? 0.0f : slab_dist(xi.z, g.lo[2] + z * g.cs, g.cs);
      if (dz * dz > rcm2) continue;
      for (int y = y0; y <= y1; ++y) {
        const float dy = g.brute ? 0.0f : slab_dist(xi.y, g.lo[1] + y * g.cs, g.cs);
        const float rem = rcm2 - dz * dz - dy * dy;
        if (rem < 0.0f) continue;
        int ja, jb;
        row_range(z, y, rem, ja, jb);
        for (int jc = ja; jc < jb; jc += L) candidate(jc + lane, jc + lane < jb);
      }
    }
  } else {
    const int ysize = y1 - y0 + 1, nrows = (z1 - z0 + 1) * ysize;
    for (int r0 = 0; r0 < nrows; r0 += L) {
      int ja = 0, jb = 0;  // of row r0 + lane
      const int r = r0 + lane;
      if (r < nrows) {
        const int z = z0 + r / ysize, y = y0 + r % ysize;
        const float dz = g.brute ? 0.0f : slab_dist(xi.z, g.lo[2] + z * g.cs, g.cs);
        const float dy = g.brute ? 0.0f : slab_dist(xi.y, g.lo[1] + y * g.cs, g.cs);
        const float rem = rcm2 - dz * dz - dy * dy;
        if (rem >= 0.0f) row_range(z, y, rem, ja, jb);
      }
      const int len = max(jb - ja, 0);
      int end = len;  // inclusive prefix over the rows
#pragma unroll
      for (int o = 1; o < L; o <<= 1) {
        const int t = __shfl_up_sync(gmask, end, o, L);
        if (lane >= o) end += t;
      }
      const int total = __shfl_sync(gmask, end, L - 1, L);
      ja -= end - len;  // candidate t of the batch is bead ja + t of its row
      for (int t0 = 0; t0 < total; t0 += L) {
        const int t = t0 + lane;
        int q = 0;  // the first row whose end lies past t
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1)
          if (__shfl_sync(gmask, end, q + o - 1, L) <= t) q += o;
        candidate(__shfl_sync(gmask, ja, q, L) + t, t < total);
      }
    }
  }
  // the list filters take entries four at a time (the stride is a multiple of 4)
  if (lane < (-cnt & 3) && cnt < stride) row[cnt + lane] = (unsigned short)(i - mstart);
  if (lane == 0) {
    s.nl_cnt[i] = cnt < stride ? cnt : (int)stride;
    if (cnt > stride) {
      atomicOr(s.flags, FLAG_NL_OVERFLOW);
      atomicMax(s.nl_maxrow, cnt);
    }
  }
}

// L lanes per bead: 8 (four beads per warp), 16 for molecules whose rows are
// long, or a warp per bead for small contexts, where fewer than a wave of
// beads leaves the latency of each bead's rounds exposed.  Beads in chain
// order: the groups of a block gather from the same region of a molecule,
// and the per-bead loads are coalesced.
template <bool UNI, int L>
__global__ void __launch_bounds__(256, 5) k_pl(DevSys s, int koff) {  // 48 registers: 5 blocks per SM
  pdl_wait();
  pdl_release();
  const int i = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) / L);
  if (i >= s.nlive) return;
  if (*s.flags & FLAG_NL_OVERFLOW) return;
  const int m = s.mol_of[i];
  if (!mol_listed(s, m, koff)) return;  // finished or stopped: keeps the lists of its last step
  int nrep, natt;
  pair_rows<UNI, L, false>(
      s, xbuf(s, m, koff), i, pair_head<L, false>(s, i, m), [](int, int) {}, [](int, float4) {}, nrep, natt);
}

// ------------------------------------------------------------ host side
static inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// Launch sequence of an exclusive scan of n ints (in -> out[0..n]).
void launch_scan(const int* in, long long n, int* out, int* block_sums, cudaStream_t st) {
  unsigned nb = cdiv(n > 0 ? n : 1, kScanTile);
  k_scan_reduce<<<nb, kScanThreads, 0, st>>>(in, n, block_sums);
  k_scan_top<<<1, 1024, 0, st>>>(block_sums, (int)nb);
  k_scan_apply<<<nb, kScanThreads, 0, st>>>(in, n, block_sums, out);
}

long long scan_block_sums_needed(long long n) { return cdiv(n > 0 ? n : 1, kScanTile) + 1; }

struct NLScratch {
  int* block_sums;
  int min_mol, max_mol;  // beads of the smallest and largest molecule the context may hold
};

// Cell binning of the molecules a rebuild at koff covers: the cell order the
// neighbour-list build walks, and each molecule's grid flags (wrap: whether
// the minimum image can matter), which the step and pair-list kernels read.
static cudaError_t launch_binning(const DevSys& s, const NLScratch& w, int koff, cudaStream_t st) {
  if (w.min_mol <= kBinMolBeads) {
    const int most = w.max_mol < kBinMolBeads ? w.max_mol : kBinMolBeads;
    const size_t sm = sizeof(int) * (3 * (size_t)most + 1);
    // a per-kernel ceiling, always the same value (contexts never lower it under
    // one another)
    const cudaError_t e = cudaFuncSetAttribute(k_bin_mol, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(int) * (3 * kBinMolBeads + 1));
    if (e != cudaSuccess) return e;
    // molecules of up to 2,048 beads take 256 threads (several blocks per SM),
    // larger ones 1,024
    const int threads = most <= 2048 ? 256 : 1024;
    k_bin_mol<<<s.nmol < 2048 ? s.nmol : 2048, threads, sm, st>>>(s, koff, most);
  }
  if (w.max_mol <= kBinMolBeads) return cudaSuccess;
  const int T = 256;
  k_bbox_reset<<<cdiv(s.nmol, T), T, 0, st>>>(s);
  k_bbox<<<cdiv(s.nlive, T), T, 0, st>>>(s, koff);
  k_grid<<<cdiv(s.nmol, T), T, 0, st>>>(s, koff);
  cudaMemsetAsync(s.cell_cnt, 0, sizeof(int) * (size_t)s.cell_cap, st);
  k_assign<<<cdiv(s.nlive, T), T, 0, st>>>(s, koff);
  launch_scan(s.cell_cnt, s.cell_cap, s.cell_scan, w.block_sums, st);
  k_scatter<<<cdiv(s.nlive, T), T, 0, st>>>(s, koff);
  k_cellsort<<<cdiv(s.cell_cap, T), T, 0, st>>>(s);
  k_stage_xs<<<cdiv(s.nlive, T), T, 0, st>>>(s, koff);
  return cudaSuccess;
}

// Full neighbour-list rebuild from the coordinates at step mol_step + koff.
void launch_nl_rebuild(const DevSys& s, const NLScratch& w, int koff, cudaStream_t st) {
  const int T = kNlThreads;
  launch_binning(s, w, koff, st);
  const bool wide = s.nlive <= kWideListBeads;
  const unsigned grid = cdiv((long long)s.nlive * (wide ? 32 : 8), T);
  if (!wide) k_att<<<cdiv(s.nlive, 128), 128, 0, st>>>(s, koff);
  if (s.uniform_type) {
    if (wide) k_nl<true, 32><<<grid, T, 0, st>>>(s, koff);
    else k_nl<true, 8><<<grid, T, 0, st>>>(s, koff);
  } else {
    if (wide) k_nl<false, 32><<<grid, T, 0, st>>>(s, koff);
    else k_nl<false, 8><<<grid, T, 0, st>>>(s, koff);
  }
}

void launch_pl_rebuild(const DevSys& s, int koff, cudaStream_t st) {
  const int T = 256;
  const int L = s.nlive <= kWideListBeads ? 32 : (s.long_rows ? 16 : 8);
  const unsigned grid = cdiv((long long)s.nlive * L, T);
  if (s.uniform_type)
    launch_pdl(L == 32 ? k_pl<true, 32> : L == 16 ? k_pl<true, 16> : k_pl<true, 8>, grid, T, st, s,
               koff);
  else
    launch_pdl(L == 32 ? k_pl<false, 32> : L == 16 ? k_pl<false, 16> : k_pl<false, 8>, grid, T, st,
               s, koff);
}

}  // namespace sop
