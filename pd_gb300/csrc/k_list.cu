// k_list.cu — cell-grid sort, blocks, tile list, exclusion masks and the
// per-evaluation position pack.  Replaces NeighbourList::calcNewList
// (PD src/mmlib/workspace/neighbourlist.cpp:222-439): PD scans all j < i at
// minimum image; here atoms are binned on a 32^3 grid ordered along a Hilbert
// curve, grouped into 32-atom blocks, and block pairs whose bounding boxes come
// within max(cutoffs)+Padding form the tile list: each row tests every column in
// systems of up to kDirectBlocks blocks, those within reach on a grid over the block
// centres in larger ones.  The bond order PD packs into
// each list entry (neighbourlist.cpp:398-422, 179-220) becomes a per-tile
// exclusion / 1-4 bit mask.
#include <algorithm>

#include <cuda_fp16.h>

#include "pdgpu_tile.cuh"
#include "pdgpu_pack.cuh"

namespace pdgpu {

// ---------------------------------------------------------------------------
// 3-D Hilbert index of a cell (J. Skilling, "Programming the Hilbert curve",
// AIP Conf. Proc. 707, 2004: axes -> transposed form, then bit interleave).
// ---------------------------------------------------------------------------
__device__ __forceinline__ int hilbert3(unsigned x0, unsigned x1, unsigned x2) {
  unsigned X[3] = {x0, x1, x2};
  const unsigned M = 1u << (kHilbertBits - 1);
  for (unsigned Q = M; Q > 1; Q >>= 1) {
    unsigned P = Q - 1;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (X[i] & Q) {
        X[0] ^= P;
      } else {
        unsigned t = (X[0] ^ X[i]) & P;
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  unsigned t = 0;
  for (unsigned Q = M; Q > 1; Q >>= 1)
    if (X[2] & Q) t ^= Q - 1;
  X[0] ^= t; X[1] ^= t; X[2] ^= t;
  int h = 0;
  for (int b = kHilbertBits - 1; b >= 0; b--) {
    h = (h << 3) | (((X[0] >> b) & 1) << 2) | (((X[1] >> b) & 1) << 1) | ((X[2] >> b) & 1);
  }
  return h;
}

// rows of systems of up to this many blocks (262,144 atoms) test every column; the tests
// grow with the square of the blocks, so larger systems take the grid.  A build of a dense
// box at R = 14 A, all columns and grid: 703 blocks 65 and 93 us, 5,623 290 and 388, 8,192
// 464 and 562, 12,288 747 and 804, 16,384 1,116 and 1,094, 24,576 1,950 and 1,586.  The two
// meet near 16,000; the line stays below, where the grid gives up 20 % at most.
constexpr int kDirectBlocks = 8192;

// order-preserving float <-> int for atomic min / max
__device__ __forceinline__ int f2ord(float f) {
  int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// What a build starts from.  The kernels of a build put these back for the next one
// once they are through with them (the first build finds them set by launch_list_init):
// cells empty, boxes of open systems turned inside out, block cells empty.
struct ListState {
  int *count, *head;               // per cell: atoms, the last of them to arrive (-1: none)
  int *lo, *hi, *hmax;             // per system, 3: box of an open system, largest half-extents
  int *bcell_count, *bcell_cursor; // per block cell
  int* counters;
  int ncells, nbcells, nsys3;
  int groups;                      // this build makes NB groups
};
__device__ __forceinline__ void reset_counter(const ListState& I, int t) {
  if (t < 8) I.counters[t] = t == 5 ? I.groups : 0;   // [5]: the NB groups fit until a row finds they do not
}
__global__ void k_list_init(ListState I, int* sorted_atom, int nslots) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
  for (int i = t; i < I.ncells; i += n) {
    I.count[i] = 0;
    I.head[i] = -1;
  }
  for (int i = t; i < nslots; i += n) sorted_atom[i] = -1;   // (padding slots keep that)
  for (int i = t; i < I.nsys3; i += n) {
    I.lo[i] = f2ord(3.0e38f);
    I.hi[i] = f2ord(-3.0e38f);
  }
}
// (a list that outgrew its arrays: its rows run again)
__global__ void k_reset_counters(ListState I) {
  pdl_sync();
  reset_counter(I, threadIdx.x);
}

// bounding box of each open-space system (periodic systems key on the box);
// a warp whose atoms share one system reduces first and adds one atomic per
// coordinate (a whole system's atoms otherwise meet on the same six words)
__global__ void k_bbox(DevView v, const int* atom_sys, int* lo, int* hi) {
  pdl_sync();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int s = a < v.natom ? atom_sys[a] : -1;
  const bool use = s >= 0 && !v.sys[s].periodic;
  const unsigned act = __ballot_sync(0xffffffffu, use);
  if (!act) return;
  const int s0 = __shfl_sync(0xffffffffu, s, __ffs(act) - 1);
  const bool uniform = __all_sync(0xffffffffu, !use || s == s0);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int x = use ? f2ord((float)v.pos[3 * a + c]) : 0;
    if (uniform) {
      int mn = use ? x : f2ord(3.0e38f), mx = use ? x : f2ord(-3.0e38f);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      }
      if (lane == __ffs(act) - 1) {
        atomicMin(&lo[3 * s0 + c], mn);
        atomicMax(&hi[3 * s0 + c], mx);
      }
    } else if (use) {
      atomicMin(&lo[3 * s + c], x);
      atomicMax(&hi[3 * s + c], x);
    }
  }
}

__device__ __forceinline__ double wrap_coord(double x, double L, double iL) { return x - L * floor(x * iL); }

// the grid of one system's block centres for this build
__device__ __forceinline__ void grid_setup(const SystemInfo& S, int s, const int* lo, const int* hi, BlockGrid* grid) {
  BlockGrid G;
  double ext[3];
  for (int c = 0; c < 3; c++) {
    if (S.periodic) {
      G.origin[c] = 0.0;
      ext[c] = S.box[c];
    } else {
      const double l = ord2f(lo[3 * s + c]), h = ord2f(hi[3 * s + c]);
      G.origin[c] = l;
      ext[c] = fmax(h - l, 1e-3);
    }
  }
  // cells of about equal edge, at most grid_cells of them
  const double edge = cbrt(ext[0] * ext[1] * ext[2] / (double)S.grid_cells);
  for (int c = 0; c < 3; c++) G.dims[c] = (int)fmax(1.0, fmin(floor(ext[c] / edge), 4096.0));
  while ((long long)G.dims[0] * G.dims[1] * G.dims[2] > S.grid_cells) {
    const int m = G.dims[0] >= G.dims[1] ? (G.dims[0] >= G.dims[2] ? 0 : 2) : (G.dims[1] >= G.dims[2] ? 1 : 2);
    G.dims[m]--;
  }
  for (int c = 0; c < 3; c++) G.cell[c] = ext[c] / G.dims[c];
  G.start = S.grid_start;
  grid[s] = G;
}

// (the last CTA, launched past the atoms where some system uses a block grid,
// sets those grids up)
__global__ void k_keys(DevView v, const int* atom_sys, ListState I, int* next, int* cell, BlockGrid* grid) {
  pdl_sync();
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  const int *lo = I.lo, *hi = I.hi;
  reset_counter(I, a);
  for (int i = a, n = gridDim.x * blockDim.x; i < max(I.nbcells, I.nsys3); i += n) {
    if (i < I.nsys3) I.hmax[i] = f2ord(0.f);
    if (i < I.nbcells) I.bcell_count[i] = I.bcell_cursor[i] = 0;
  }
  if (grid && blockIdx.x == gridDim.x - 1) {
    for (int s = threadIdx.x; s < v.nsys; s += blockDim.x)
      if (v.sys[s].nblocks > kDirectBlocks) grid_setup(v.sys[s], s, lo, hi, grid);
    return;
  }
  if (a >= v.natom) return;
  int s = atom_sys[a];
  const SystemInfo& S = v.sys[s];
  unsigned q[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    double x = v.pos[3 * a + c];
    double f;
    if (S.periodic) {
      f = wrap_coord(x, S.box[c], S.ibox[c]) * S.ibox[c];
    } else {
      double l = ord2f(lo[3 * s + c]), h = ord2f(hi[3 * s + c]);
      f = (x - l) / (h - l + 1e-3);
    }
    int qi = (int)(f * (1 << kHilbertBits));
    qi = qi < 0 ? 0 : (qi > (1 << kHilbertBits) - 1 ? (1 << kHilbertBits) - 1 : qi);
    q[c] = (unsigned)qi;
  }
  int b = s * kCellsPerSystem + hilbert3(q[0], q[1], q[2]);
  cell[a] = b;
  next[a] = atomicExch(&I.head[b], a);
  atomicAdd(&I.count[b], 1);
}

// --- exclusive scans --------------------------------------------------------
__device__ __forceinline__ int warp_inclusive_scan(int x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// 1024 threads: the exclusive prefix of each thread's value within the CTA
// (warp scans, then a scan of the 32 warp totals); *total gets the CTA's sum
__device__ __forceinline__ int cta_exclusive_scan(int x, int* wsum, int* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int inc = warp_inclusive_scan(x, lane);
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const int t = wsum[lane];
    const int ti = warp_inclusive_scan(t, lane);
    wsum[lane] = ti - t;
    if (lane == 31) wsum[32] = ti;
  }
  __syncthreads();
  *total = wsum[32];
  return wsum[wid] + inc - x;
}

// two-phase scan, 1024 elements per CTA
__global__ void __launch_bounds__(1024) k_scan_block(const int* in, int* out, int* block_sums, int n) {
  pdl_sync();
  __shared__ int wsum[33];
  const int i = blockIdx.x * 1024 + threadIdx.x;
  const int x = i < n ? in[i] : 0;
  int total;
  const int e = cta_exclusive_scan(x, wsum, &total);
  if (i < n) out[i] = e;
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// each CTA sums the totals before its own and adds them
__global__ void __launch_bounds__(1024) k_scan_add(int* out, const int* sums, int n) {
  pdl_sync();
  __shared__ int wsum[33];
  int before = 0;
  for (int i = threadIdx.x; i < blockIdx.x; i += 1024) before += sums[i];
  int total;
  cta_exclusive_scan(before, wsum, &total);
  const int i = blockIdx.x * 1024 + threadIdx.x;
  if (i < n) out[i] += total;
}

// one CTA for n <= kScanOne: 8 consecutive elements per thread
constexpr int kScanOne = 8192;
__global__ void __launch_bounds__(1024) k_scan_one(const int* in, int* out, int n) {
  pdl_sync();
  __shared__ int wsum[33];
  const int base = threadIdx.x * 8;
  int x[8], s = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    x[k] = base + k < n ? in[base + k] : 0;
    s += x[k];
  }
  int total;
  int run = cta_exclusive_scan(s, wsum, &total);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (base + k < n) out[base + k] = run;
    run += x[k];
  }
}

// A thread per cell: the cell's place (after the system's atoms in runs of 1024 cells
// before, whose sums k_scan_block left with the cells' offsets within their runs), its
// atoms from their chain, in ascending order so that the result is deterministic, into
// their slots.  The chain runs from the last atom to arrive to the first, near enough
// descending: it is inserted from the end of the cell's run, where few have to move.
// A crowded cell would keep its one thread busy for long (a chain is a load after the
// other, and insertion grows with the square of what arrived out of order): one atom far
// away from an open system, or coordinates that are not finite, put all others into one.
// The CTA places the atoms of such cells together: its warps walk the system's atoms in
// ascending order, each an eighth of them, and count, then place, those of its crowded
// cells.  A walk costs some 2 x natom / 256 loads in a row, a chain one load an atom and
// the insertion on top, so cells count as crowded from natom / 512 atoms on, within the
// bounds below (a dense box of the largest size has 64 atoms a cell).  A build of an open
// system of 3,000 atoms with one of them far away: 104 ms with each cell sorted by its
// thread in order of arrival, 50 us so (39 us without that atom); 30,000 atoms 262 us.
constexpr int kSortThreads = 256;
constexpr int kCrowdedMin = 64, kCrowdedMax = 512;
__device__ __forceinline__ int warp_sum_int(int x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
// the atoms of the CTA's crowded cells into their slots (place: each such cell's first
// slot, -1 for the others); every thread of the CTA calls this
__device__ __forceinline__ void place_crowded(const SystemInfo& S, const int* cell, const int* place, int (*cur)[kSortThreads],
                                              int* sorted_atom, int* slot_of) {
  constexpr int W = kSortThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = blockIdx.x * kSortThreads;
  const unsigned lt = (1u << lane) - 1u;
  const int per = (S.natom + W - 1) / W;
  const int a0 = S.atom_start + min(wid * per, S.natom), a1 = S.atom_start + min((wid + 1) * per, S.natom);
  for (int w = 0; w < W; w++) cur[w][threadIdx.x] = 0;
  __syncthreads();
  for (int pass = 0; pass < 2; pass++) {
#pragma unroll 4
    for (int i = a0; i < a1; i += 32) {
      const int a = i + lane, c = a < a1 ? cell[a] - c0 : -1;
      const bool mine = c >= 0 && c < kSortThreads && place[c] >= 0;
      if (!__any_sync(0xffffffffu, mine)) continue;
      const unsigned m = __match_any_sync(0xffffffffu, mine ? c : -1);
      if (mine && pass) {
        const int s = cur[wid][c] + __popc(m & lt);
        sorted_atom[s] = a;
        slot_of[a] = s;
      }
      __syncwarp();
      if (mine && !(m & lt)) cur[wid][c] += __popc(m);
      __syncwarp();
    }
    __syncthreads();
    if (pass == 0) {   // counts to each warp's first slot of each cell
      int s = place[threadIdx.x];
      for (int w = 0; w < W; w++) {
        const int n = cur[w][threadIdx.x];
        cur[w][threadIdx.x] = s;
        s += n;
      }
      __syncthreads();
    }
  }
}
__global__ void __launch_bounds__(kSortThreads) k_cell_sort(DevView v, ListState I, const int* offset, const int* run_sums,
                                                            const int* next, const int* cell, int* tmp, int* sorted_atom,
                                                            int* slot_of) {
  static_assert(kCellsPerSystem == 32 * 1024 && 1024 % kSortThreads == 0, "a warp adds a system's runs");
  pdl_sync();
  __shared__ int base, place[kSortThreads], cur[kSortThreads / 32][kSortThreads];
  const int b = blockIdx.x * kSortThreads + threadIdx.x;   // (ncells is a multiple of 1024)
  const SystemInfo& S = v.sys[b / kCellsPerSystem];
  if (threadIdx.x < 32) {
    const int run = b / 1024, r0 = b / kCellsPerSystem * 32;
    const int x = warp_sum_int(r0 + (int)threadIdx.x < run ? run_sums[r0 + threadIdx.x] : 0);
    if (threadIdx.x == 0) base = S.atom_start + x;
  }
  const int n = I.count[b];
  int a = n ? I.head[b] : -1;
  __syncthreads();
  const int o = base + (n ? offset[b] : 0);
  if (b < I.nsys3) {
    I.lo[b] = f2ord(3.0e38f);
    I.hi[b] = f2ord(-3.0e38f);
  }
  if (n > 0) {
    I.count[b] = 0;
    I.head[b] = -1;
  }
  const int slot = S.pad_start + (o - S.atom_start);
  const bool crowded = n > min(max(S.natom / 512, kCrowdedMin), kCrowdedMax);
  place[threadIdx.x] = crowded ? slot : -1;
  if (__syncthreads_or(crowded)) place_crowded(S, cell, place, cur, sorted_atom, slot_of);
  if (n < 1 || crowded) return;
  int* p = tmp + o;
  for (int i = n - 1; i >= 0; i--) {
    const int x = a;
    a = next[a];
    int j = i + 1;
    while (j < n && p[j] < x) {
      p[j - 1] = p[j];
      j++;
    }
    p[j - 1] = x;
  }
  for (int i = 0; i < n; i++) {
    const int x = p[i];
    sorted_atom[slot + i] = x;
    slot_of[x] = slot + i;
  }
}

// cell coordinate of x along axis c (clamped into the grid)
__device__ __forceinline__ int grid_axis(const BlockGrid& G, int c, double x) {
  const double q = floor((x - G.origin[c]) / G.cell[c]);
  return (int)fmin(fmax(q, 0.0), (double)(G.dims[c] - 1));
}

// One warp per block: its box (centre and half-extents), its slots' parameters and
// packed positions, and its cell where the system's rows use the block grid.  FP32
// box arithmetic with the half-extents on the safe side; the centre is an FP32
// number, so that centre differences are exact in double-float arithmetic.
struct SlotParams {
  const double *radius, *sqeps, *gbR, *gbVj, *lcR, *charge;
  const int* lcUse;
  float4* lc_par;
};
__device__ __forceinline__ void slot_params(const DevView& v, const SlotParams& P, int s, int a) {
  float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 l = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a >= 0) {
    p.x = (float)P.radius[a];
    p.y = (float)P.sqeps[a];
    if (P.gbR) {
      p.z = (float)P.gbR[a];
      p.w = (float)P.gbVj[a];
    }
    if (P.lcR) {
      l.x = (float)P.lcR[a];
      l.y = P.lcUse[a] ? 1.f : 0.f;
    }
  }
  v.par[s] = p;
  if (P.lc_par) P.lc_par[s] = l;
}

__global__ void __launch_bounds__(128) k_blocks(DevView v, SlotParams P, StepClear C, const BlockGrid* grid, int* hmax,
                                                int* bcell, int* bcount, int sub) {
  pdl_sync();
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= v.nblocks) return;
  const int slot = b * 32 + lane;
  const int a = v.sorted_atom[slot];
  const int sys = v.slot_sys[b];
  const SystemInfo& S = v.sys[sys];
  float lo[3], hi[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    double x = 0;
    if (a >= 0) {
      x = v.pos[3 * a + c];
      if (S.periodic) x = wrap_coord(x, S.box[c], S.ibox[c]);
    }
    lo[c] = a >= 0 ? (float)x : 3.0e38f;
    hi[c] = a >= 0 ? (float)x : -3.0e38f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
  }
  slot_params(v, P, slot, a);
  step_clear(C, v, slot);
  float cf[3], hf[3];
  double cd[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    cf[c] = 0.5f * lo[c] + 0.5f * hi[c];
    cd[c] = (double)cf[c];
    hf[c] = fmaxf(hi[c] - cf[c], cf[c] - lo[c]) + 1e-4f + 2.4e-7f * fmaxf(fabsf(lo[c]), fabsf(hi[c]));
  }
  const float4 o = packed_slot(v, S, P.charge, slot, a, v.pos + 3 * (a < 0 ? 0 : a), cd);
  v.xq[slot] = o;
  v.rel0[slot] = o;
  if (sub) write_sub(v, slot, o);
  if (P.gbR) write_radius(v, slot, a, o);
  if (lane == 0) {
    v.half[b] = make_float4(hf[0], hf[1], hf[2], 0.f);
    v.cenf[b] = make_float4(cf[0], cf[1], cf[2], 0.f);
#pragma unroll
    for (int c = 0; c < 3; c++) v.center[3 * b + c] = cd[c];
    if (S.nblocks > kDirectBlocks) {
      const BlockGrid& G = grid[sys];
      const int cell = G.start + (grid_axis(G, 2, cd[2]) * G.dims[1] + grid_axis(G, 1, cd[1])) * G.dims[0] +
                       grid_axis(G, 0, cd[0]);
      bcell[b] = cell;
      atomicAdd(&bcount[cell], 1);
#pragma unroll
      for (int c = 0; c < 3; c++) atomicMax(&hmax[3 * sys + c], f2ord(hf[c]));
    }
  }
}
// static per-slot parameters (LJ radius, sqrt eps, GB radius, Vj) after a parameter update
__global__ void k_slot_params(DevView v, SlotParams P) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < v.nslots) slot_params(v, P, s, v.sorted_atom[s]);
}

// ---------------------------------------------------------------------------
// Tile list.  Block pair (bi, bj), bi <= bj of one system, is a tile when the
// two blocks' bounding boxes come within R (periodic: at the minimum image of
// their centres).  One CTA per row bi finds the row's hits in a bitmap over its
// columns bj >= bi, takes its place in the list with one atomic on the tile total
// and writes its tiles there in ascending bj.  Rows land in any order, each
// contiguous with ascending columns (what the work items and the NB groups rely
// on); every sum over tiles is in fixed point, so the results do not depend on the
// rows' order.
//  * Systems of up to kDirectBlocks blocks test every column (32 per warp step).
//  * Larger ones bin their block centres on a grid of at most one cell per block;
//    a row visits only the cells within R + h_i + hmax of its centre along each
//    axis (h: half-extents, hmax the system's largest), so the work follows the
//    tiles, not the square of the block count.
// The tiles that need exclusion bits (diagonal, a system's padded last block, a
// bonded pair) are marked in a second bitmap from the row's atoms' partners and go
// to a list as they are written.
// ---------------------------------------------------------------------------
// box test of one block pair; flags as Tile::flags.  FP32 geometry (the FP64
// pipe is narrow on this GPU), every decision taken 1e-3 A on the safe side:
// include, per-pair image, not all-inside
__device__ __forceinline__ bool tile_test(const DevView& v, const SystemInfo& S, int gi, int gj, float R,
                                          float margin, float full_R, float full_margin, int& flags) {
  const float4 hi4 = v.half[gi], hj4 = v.half[gj];
  const float hs[3] = {hi4.x + hj4.x, hi4.y + hj4.y, hi4.z + hj4.z};
  const float4 ci4 = v.cenf[gi], cj4 = v.cenf[gj];
  const float ci[3] = {ci4.x, ci4.y, ci4.z}, cj[3] = {cj4.x, cj4.y, cj4.z};
  constexpr float kSafe = 1e-3f;
  float dist2 = 0.f, dmax2 = 0.f;
  bool need_mi = false;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    float d = cj[c] - ci[c];
    if (S.periodic) {
      const float L = S.boxf[c].h;
      d -= L * rintf(d / L);
      // a pair of the two blocks inside the cutoff in some other image would
      // sit at least L - R apart along this axis in the tile's image: below
      // that every pair inside the cutoff takes the tile's image, and pairs
      // whose images differ lie beyond the cutoff in both
      if (fabsf(d) + hs[c] + margin >= L - R - kSafe) need_mi = true;
    }
    const float g = fabsf(d) - hs[c];
    if (g > 0.f) dist2 += g * g;
    const float m = fabsf(d) + hs[c];
    dmax2 += m * m;
  }
  // full: the farthest pair of the two boxes, grown by the displacement margin,
  // stays inside every cutoff and switch radius
  const bool full = full_R > 0.f && !need_mi && sqrtf(dmax2) + full_margin + kSafe < full_R;
  flags = (need_mi ? 1 : 0) | (gi == gj ? 2 : 0) | (full ? 4 : 0);
  const float Rs = R + kSafe;
  return dist2 <= Rs * Rs;
}

// the tile record at position t (centre offset formed in FP64, rounded once)
__device__ __forceinline__ void write_tile(const DevView& v, const SystemInfo& S, int gi, int gj, int flags,
                                           long long t, long long cap) {
  if (t >= cap) return;
  Tile T;
  T.bi = gi;
  T.bj = gj;
  T.mask = -1;
  T.flags = flags;
  double o[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    o[c] = v.center[3 * gj + c] - v.center[3 * gi + c];
    if (S.periodic) o[c] -= S.box[c] * rint(o[c] * S.ibox[c]);
  }
  T.ox = (float)o[0];
  T.oy = (float)o[1];
  T.oz = (float)o[2];
  T.pad = 0.f;
  v.tiles[t] = T;
}

// blocks in cell order (the order inside a cell does not matter: rows collect
// their hits in a bitmap)
__global__ void k_bgrid_scatter(DevView v, const int* bcell, const int* offset, int* cursor, int* blocks) {
  pdl_sync();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= v.nblocks || v.sys[v.slot_sys[b]].nblocks <= kDirectBlocks) return;
  const int cell = bcell[b];
  blocks[offset[cell] + atomicAdd(&cursor[cell], 1)] = b;
}

// position of the n-th (from 0) set bit of m (m holds more than n set bits)
__device__ __forceinline__ int nth_set_bit(unsigned m, int n) {
  int pos = 0;
#pragma unroll
  for (int b = 16; b > 0; b >>= 1) {
    const int c = __popc(m & ((1u << b) - 1u));
    if (n >= c) {
      n -= c;
      m >>= b;
      pos += b;
    }
  }
  return pos;
}

constexpr int kRowWarps = 4;
// marks the row's tiles that hold a bonded pair: each atom of block bi, its
// partners of either side (band words, far list); the warps take one kind each
__device__ __forceinline__ void mark_partner(const int* slot_of, int bi, int nw, const unsigned* bits, unsigned* mbits,
                                             int b) {
  const int o = (slot_of[b] >> 5) - bi;
  if (o <= 0 || (o >> 5) >= nw) return;   // (the diagonal is marked anyway; lower rows mark their own)
  if ((bits[o >> 5] >> (o & 31)) & 1u) atomicOr(&mbits[o >> 5], 1u << (o & 31));
}

// `words` words of either bitmap in dynamic shared memory; positions past `cap`
// are dropped (k_masks flags the overflow)
__global__ void __launch_bounds__(kRowWarps * 32) k_tile_rows(DevView v, const BlockGrid* grid, const int* hmax,
                                                              const int* cell_off, const int* cell_count,
                                                              const int* cell_blocks, const int* slot_of, float R,
                                                              float margin, float full_R, float full_margin,
                                                              int* row_cnt, int* row_start, long long cap, int words,
                                                              int* total, int* mlist, int* nml) {
  pdl_sync();
  extern __shared__ unsigned s_bits[];
  __shared__ int s_cnt[kRowWarps], s_base;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, bi = blockIdx.x;
  unsigned *bits = s_bits, *mbits = s_bits + words;
  const int sys = v.slot_sys[bi];
  const SystemInfo& S = v.sys[sys];
  const int end = S.block_start + S.nblocks;
  const int nw = (end - bi + 31) >> 5;
  if (S.nblocks <= kDirectBlocks) {
    for (int w = wid; w < nw; w += kRowWarps) {
      const int bj = bi + 32 * w + lane;
      int fl = 0;
      const unsigned m = __ballot_sync(0xffffffffu, bj < end && tile_test(v, S, bi, bj, R, margin, 0.f, 0.f, fl));
      if (lane == 0) {
        bits[w] = m;
        mbits[w] = w == 0 ? 1u : 0u;   // the diagonal
      }
    }
    __syncthreads();
  } else {
    const BlockGrid& G = grid[sys];
    const float4 h4 = v.half[bi];
    const float h[3] = {h4.x, h4.y, h4.z};
    for (int w = threadIdx.x; w < nw; w += kRowWarps * 32) {
      bits[w] = 0u;
      mbits[w] = w == 0 ? 1u : 0u;
    }
    __syncthreads();
    int lo[3], hi[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double x = v.center[3 * bi + c] - G.origin[c];
      // reach along the axis: list radius, both half-extents, and a slack far
      // above the rounding of the centres and cell edges
      const double r = (double)R + (double)h[c] + (double)ord2f(hmax[3 * sys + c]) + 0.01;
      const int D = G.dims[c];
      int a = (int)fmax(floor((x - r) / G.cell[c]), -1.0e9);
      int b = (int)fmin(floor((x + r) / G.cell[c]), 1.0e9);
      if (S.periodic) {
        if (b - a + 1 >= D) {
          a = 0;
          b = D - 1;
        }
      } else {
        a = max(a, 0);
        b = min(b, D - 1);
      }
      lo[c] = a;
      hi[c] = b;
    }
    // the cell runs to visit: one per (y, z) cell row of the range, two where
    // a periodic x range wraps, dealt over the warps.  Each lane reads one run's
    // block range, then the warp deals the runs' blocks over its lanes (the reads
    // of a row are independent of one another, not a chain of dependent loads)
    const int Dx = G.dims[0], Dy = G.dims[1], Dz = G.dims[2];
    const int nyr = hi[1] - lo[1] + 1, nzr = hi[2] - lo[2] + 1;
    const bool wrapx = lo[0] < 0 || hi[0] >= Dx;
    const int nxr = wrapx ? 2 : 1;
    const int nrun = nyr * nzr * nxr;
    for (int q0 = 0; q0 < nrun; q0 += 32 * kRowWarps) {
      const int q = q0 + lane * kRowWarps + wid;
      int p0 = 0, len = 0;
      if (q < nrun) {
        const int xr = q % nxr, yz = q / nxr;
        const int cy = ((lo[1] + yz % nyr) % Dy + Dy) % Dy, cz = ((lo[2] + yz / nyr) % Dz + Dz) % Dz;
        const int row0 = G.start + (cz * Dy + cy) * Dx;
        int c0 = lo[0], c1 = hi[0];
        if (lo[0] < 0) {
          c0 = xr ? 0 : lo[0] + Dx;
          c1 = xr ? hi[0] : Dx - 1;
        } else if (hi[0] >= Dx) {
          c0 = xr ? 0 : lo[0];
          c1 = xr ? hi[0] - Dx : Dx - 1;
        }
        p0 = cell_off[row0 + c0];
        len = cell_off[row0 + c1] + cell_count[row0 + c1] - p0;
      }
      const int inc = warp_inclusive_scan(len, lane);
      const int cnt = __shfl_sync(0xffffffffu, inc, 31);
      const int excl = inc - len;
      for (int t0 = 0; t0 < cnt; t0 += 32) {
        const int t = t0 + lane;
        // the run holding entry t: the last lane whose runs start at or before t
        int L = 0;
#pragma unroll
        for (int b = 16; b > 0; b >>= 1)
          if (__shfl_sync(0xffffffffu, excl, L + b) <= t) L += b;
        const int p = __shfl_sync(0xffffffffu, p0, L) + t - __shfl_sync(0xffffffffu, excl, L);
        if (t < cnt) {
          const int bj = cell_blocks[p];
          int fl;
          if (bj >= bi && tile_test(v, S, bi, bj, R, margin, 0.f, 0.f, fl))
            atomicOr(&bits[(bj - bi) >> 5], 1u << ((bj - bi) & 31));
        }
      }
    }
    __syncthreads();
  }
  // tiles that get an exclusion mask
  const int a = v.sorted_atom[bi * 32 + lane];
  if (a >= 0) {
    if (wid == 0) {
      for (unsigned long long m = v.band_excl[a] | v.band_14[a]; m; m &= m - 1)
        mark_partner(slot_of, bi, nw, bits, mbits, a + __ffsll((long long)m));
    } else if (wid == 1) {
      for (unsigned long long m = v.band_dn_excl[a] | v.band_dn_14[a]; m; m &= m - 1)
        mark_partner(slot_of, bi, nw, bits, mbits, a - __ffsll((long long)m));
    } else if (wid == 2) {
      for (int q = v.far_both_start[a]; q < v.far_both_start[a + 1]; q++)
        mark_partner(slot_of, bi, nw, bits, mbits, v.far_both_idx[q]);
    }
  }
  if (threadIdx.x == kRowWarps * 32 - 1 && S.natom != S.npad) {   // the system's padded last block
    const int o = end - 1 - bi;
    if ((bits[o >> 5] >> (o & 31)) & 1u) atomicOr(&mbits[o >> 5], 1u << (o & 31));
  }
  // each warp writes a run of the words; the row's place by one atomic
  const int per = (nw + kRowWarps - 1) / kRowWarps;
  const int wa = min(wid * per, nw), wb = min(wa + per, nw);
  int k = 0;
  for (int w = wa + lane; w < wb; w += 32) k += __popc(bits[w]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
  if (lane == 0) s_cnt[wid] = k;
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int w = 0; w < kRowWarps; w++) n += s_cnt[w];
    s_base = atomicAdd(total, n);
    row_start[bi] = s_base;
    row_cnt[bi] = n;
  }
  __syncthreads();
  long long base = s_base;
  for (int w = 0; w < wid; w++) base += s_cnt[w];
  for (int w0 = wa; w0 < wb; w0 += 32) {
    const int w = w0 + lane;
    const unsigned word = w < wb ? bits[w] : 0u;
    const int kw = __popc(word);
    const int inc = warp_inclusive_scan(kw, lane);
    const int tot = __shfl_sync(0xffffffffu, inc, 31);
    // the hits of these 32 words dealt over the lanes, in column order
    const int excl = inc - kw;
    for (int t0 = 0; t0 < tot; t0 += 32) {
      const int t = t0 + lane;
      int L = 0;
#pragma unroll
      for (int b = 16; b > 0; b >>= 1)
        if (__shfl_sync(0xffffffffu, excl, L + b) <= t) L += b;
      const unsigned wl = __shfl_sync(0xffffffffu, word, L);
      const int nth = t - __shfl_sync(0xffffffffu, excl, L);
      if (t < tot) {
        const int bit = nth_set_bit(wl, nth);
        const int bj = bi + 32 * (w0 + L) + bit;
        int fl = 0;
        tile_test(v, S, bi, bj, R, margin, full_R, full_margin, fl);
        write_tile(v, S, bi, bj, fl, base + t, cap);
        if (base + t < cap && ((mbits[w0 + L] >> bit) & 1u)) {
          const int q = atomicAdd(nml, 1);
          if (q < v.mask_cap) mlist[q] = (int)(base + t);
        }
      }
    }
    base += tot;
  }
}

// one warp per tile of the mask list (grid-stride): the tile's exclusion and
// 1-4 bits, a mask table entry when any is set.  Each lane walks its i atom's own
// bonded partners of either side (a few) and looks up their slots; asking each of the
// tile's 32 j atoms for its bond instead took 9, 13 and 45 us at 2,001, 22,489 and
// 179,912 atoms.
// (also the tile count from the rows' total, clamped to the capacity: an overflow
// leaves a short list and is flagged)
__global__ void k_masks(DevView v, const int* slot_of, const int* mlist, const int* nml, const int* total, long long cap) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const int n = min(*nml, v.mask_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const long long t = *total;
    *v.ntiles = (int)(t < cap ? t : cap);
    if (t > cap) atomicOr(v.status, (unsigned)ST_TILE_OVERFLOW);
  }
  if (*nml > v.mask_cap && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(v.status, (unsigned)ST_TILE_OVERFLOW);
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < n; e += nwarps) {
    const int warp = mlist[e];
    Tile T = v.tiles[warp];
    const int ai = v.sorted_atom[T.bi * 32 + lane];
    // bit k of a lane stands for the j atom k slots on, around the block; padding
    // slots, and a diagonal tile's own atom, are excluded
    const unsigned pad = __ballot_sync(0xffffffffu, v.sorted_atom[T.bj * 32 + lane] < 0);
    unsigned ex = __funnelshift_r(pad, pad, lane) | (T.bi == T.bj ? 1u : 0u), m14 = 0u;
    if (ai < 0) {
      ex = 0xffffffffu;
    } else {
      auto partner = [&](int a, bool excluded) {
        const int s = slot_of[a];
        if ((s >> 5) != T.bj) return;
        const unsigned bit = 1u << ((s - lane) & 31);
        if (excluded) ex |= bit;
        else m14 |= bit;
      };
      const unsigned long long xu = v.band_excl[ai], xd = v.band_dn_excl[ai];
      for (unsigned long long m = xu | v.band_14[ai]; m; m &= m - 1)
        partner(ai + __ffsll((long long)m), xu & m & (~m + 1));
      for (unsigned long long m = xd | v.band_dn_14[ai]; m; m &= m - 1)
        partner(ai - __ffsll((long long)m), xd & m & (~m + 1));
      for (int q = v.far_both_start[ai]; q < v.far_both_start[ai + 1]; q++)
        if (v.far_both_bo[q] <= 3) partner(v.far_both_idx[q], v.far_both_bo[q] <= 2);
      m14 &= ~ex;
    }
    bool any = __any_sync(0xffffffffu, (ex | m14) != 0);
    if (!any) continue;
    int idx = 0;
    if (lane == 0) idx = atomicAdd(v.nmasks, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= v.mask_cap) {
      // (the capacity bounds the diagonal, padded and bonded tiles: not reached)
      if (lane == 0) atomicOr(v.status, (unsigned)ST_TILE_OVERFLOW);
      continue;
    }
    v.masks[idx * 32 + lane] = make_uint2(ex, m14);
    if (lane == 0) v.tiles[warp].mask = idx;
  }
}

// per-evaluation pack (between list builds): the slots at the current positions
__global__ void k_pack(DevView v, PackArgs P) {
  pdl_sync();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= v.nslots) return;   // (whole warps)
  const int a = v.sorted_atom[s];
  pack_slot(v, P, s, a, v.pos + 3 * (a < 0 ? 0 : a));
}

// GB work items, one warp per row: the row's all-inside tiles without exclusion
// mask (far: where the passes find all-inside tiles at run time, every tile
// without one) go together two by two in column order (a pairing that does not depend on
// the other systems of a batch), every other tile is an item of its own; the row's
// items take their place by an atomic on the total (any order: every sum is in
// fixed point).  pairs: 0 makes every item a single tile
__global__ void __launch_bounds__(128) k_items(DevView v, int pairs, int far, const int* row_start, const int* row_cnt) {
  pdl_sync();
  const int lane = threadIdx.x & 31, b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (b >= v.nblocks) return;
  const int t0 = row_start[b], n = max(min(row_cnt[b], *v.ntiles - t0), 0);
  int np = 0;
  for (int i = 0; i < n; i += 32) {
    bool p = false;
    if (pairs && i + lane < n) {
      const Tile T = v.tiles[t0 + i + lane];
      p = (far || tile_full(T)) && !tile_masked(T) && !(T.flags & 1);
    }
    np += __popc(__ballot_sync(0xffffffffu, p));
  }
  int base = 0;
  if (lane == 0) base = atomicAdd(v.nitems, (np + 1) / 2 + n - np);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (lane == 0 && (np & 1)) v.items[base + np / 2].y = -1;   // the last one stays alone
  int* two = reinterpret_cast<int*>(v.items + base);
  int2* one = v.items + base + (np + 1) / 2;
  int rp = 0, rs = 0;
  const unsigned lt = (1u << lane) - 1u;
  for (int i = 0; i < n; i += 32) {
    const bool in = i + lane < n;
    bool p = false;
    if (pairs && in) {
      const Tile T = v.tiles[t0 + i + lane];
      p = (far || tile_full(T)) && !tile_masked(T) && !(T.flags & 1);
    }
    const unsigned mp = __ballot_sync(0xffffffffu, p), ms = __ballot_sync(0xffffffffu, in && !p);
    if (p) two[rp + __popc(mp & lt)] = t0 + i + lane;
    else if (in) one[rs + __popc(ms & lt)] = make_int2(t0 + i + lane, -1);
    rp += __popc(mp);
    rs += __popc(ms);
  }
}

// ---------------------------------------------------------------------------
// NB j-atom groups.  A 32x32 tile at list radius R holds ~12 % pairs inside a
// 12 A cutoff (dense solvent, 7.5 A blocks); most of its j atoms lie beyond R
// of the whole i block.  Per i-block row, the j atoms of the row's plain tiles
// (no exclusion mask, off-diagonal, one periodic image) that lie within R of the
// i block's box are packed into groups of 32; the pair kernel rotates a group
// like a tile's j block.  Valid while every atom stays within half the skin of
// its build position (the per-step displacement check, forced on with groups):
// a pair inside the cutoff then had its j atom within R of the i box at build.
// The row's j atoms go by class: which of the block's four 8-atom sub-blocks lie
// within the cutoffs of the atom, in Gray-code order, so that a group's atoms reach
// the same sub-blocks and the force pass skips the others; those in the skin alone
// (no sub-block) come last.  Sorted this way a solvated box of 22,489 atoms at 12 A
// computes 2.2 pairs per pair inside the cutoff instead of 3.0 (within the cutoffs
// first, then the skin) and 4.4 (unskipped).  One CTA per row: its warps take
// consecutive runs of the row's tiles, count, take the row's groups by an atomic on
// the total (rows in any order: every sum is in fixed point) and write; a class keeps
// tile order, then lane order.  A row's groups are an even number (the force pass
// takes two at once).
// ---------------------------------------------------------------------------
constexpr int kCullClasses = 16;
// class c holds the atoms that reach the sub-blocks of Gray code c + 1 (the last: none)
__device__ __forceinline__ unsigned cull_code(int c) {
  const unsigned g = (c + 1) & 15;
  return g ^ (g >> 1);
}
__device__ __forceinline__ int cull_class(unsigned code) {
  return ((code ^ (code >> 1) ^ (code >> 2) ^ (code >> 3)) + 15) & 15;
}
// lanes of a tile whose j atom has the given code: r[s] those that reach sub-block s,
// of the kept ones
__device__ __forceinline__ unsigned cull_lanes(unsigned code, const uint4& r, unsigned kept) {
  const unsigned a = (code & 1u) - 1u, b = ((code >> 1) & 1u) - 1u, c = ((code >> 2) & 1u) - 1u, d = ((code >> 3) & 1u) - 1u;
  return kept & (r.x ^ a) & (r.y ^ b) & (r.z ^ c) & (r.w ^ d);
}

// what pass one leaves of a tile: the lanes that reach each sub-block, the lanes kept,
// whether the tile stays a tile
struct __align__(16) CullTile {
  uint4 r;
  unsigned kept, rest, pad[2];
};

// W: warps of a row's CTA.  16 while a row's latency counts (fewer than 8 rows an SM:
// 703 rows 37 -> 24 us), 8 above (5,623 rows: 16 warps are 14 us slower)
template <int W>
__global__ void __launch_bounds__(W * 32, 48 / W) k_cull(DevView v, float R2, float Rc2, const int* row_start, const int* row_cnt,
                                                 CullTile* info) {
  pdl_sync();
  // the sub-blocks' boxes two by two: centres, half-extents.  FP16 is ample to sort
  // atoms into classes (0.01 A at 16 A): the force pass tests the boxes itself.
  __shared__ __half2 sc[2][3], sh[2][3];
  __shared__ int cnt[W][kCullClasses + 1];   // per class; [kCullClasses]: tiles that stay tiles
  __shared__ int first, first_rest;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, b = blockIdx.x;
  const int t0 = row_start[b], n = min(row_cnt[b], *v.ntiles - t0);
  const int per = (max(n, 0) + W - 1) / W;
  const int ta = t0 + min(wid * per, max(n, 0)), tb = t0 + min((wid + 1) * per, max(n, 0));
  const float4 h = v.half[b];
  const SystemInfo& S = v.sys[v.slot_sys[b]];
  const int last = S.block_start + S.nblocks - 1;   // the block that holds the system's padding slots
  if (threadIdx.x < 2) {
    const float4 l0 = v.sub[8 * b + 4 * threadIdx.x], h0 = v.sub[8 * b + 4 * threadIdx.x + 1];
    const float4 l1 = v.sub[8 * b + 4 * threadIdx.x + 2], h1 = v.sub[8 * b + 4 * threadIdx.x + 3];
    sc[threadIdx.x][0] = __floats2half2_rn(0.5f * (l0.x + h0.x), 0.5f * (l1.x + h1.x));
    sc[threadIdx.x][1] = __floats2half2_rn(0.5f * (l0.y + h0.y), 0.5f * (l1.y + h1.y));
    sc[threadIdx.x][2] = __floats2half2_rn(0.5f * (l0.z + h0.z), 0.5f * (l1.z + h1.z));
    sh[threadIdx.x][0] = __floats2half2_rn(0.5f * (h0.x - l0.x), 0.5f * (h1.x - l1.x));
    sh[threadIdx.x][1] = __floats2half2_rn(0.5f * (h0.y - l0.y), 0.5f * (h1.y - l1.y));
    sh[threadIdx.x][2] = __floats2half2_rn(0.5f * (h0.z - l0.z), 0.5f * (h1.z - l1.z));
  }
  __syncthreads();
  __half2 C[2][3], H[2][3];
#pragma unroll
  for (int q = 0; q < 2; q++)
#pragma unroll
    for (int k = 0; k < 3; k++) {
      C[q][k] = sc[q][k];
      H[q][k] = sh[q][k];
    }
  const __half2 zero = __float2half2_rn(0.f), rc2 = __float2half2_rn(Rc2);
  const unsigned mine = cull_code(lane & 15);   // lanes 0-15 keep the counts of a class each
  int mycnt = 0, rest = 0;
#pragma unroll 1
  for (int t = ta; t < tb; t++) {
    const Tile T = v.tiles[t];
    const bool plain = T.mask < 0 && !(T.flags & 3);
    const int sj = T.bj * 32 + lane;
    float4 x = v.xq[sj];
    x.x += T.ox;
    x.y += T.oy;
    x.z += T.oz;
    const float gx = fmaxf(fabsf(x.x) - h.x, 0.f), gy = fmaxf(fabsf(x.y) - h.y, 0.f);
    const float gz = fmaxf(fabsf(x.z) - h.z, 0.f);
    const bool keep = plain && gx * gx + gy * gy + gz * gz <= R2 && (T.bj != last || v.sorted_atom[sj] >= 0);
    const unsigned kept = __ballot_sync(0xffffffffu, keep);
    rest += plain ? 0 : 1;
    CullTile I;
    I.r = make_uint4(0u, 0u, 0u, 0u);
    I.kept = kept;
    I.rest = plain ? 0u : 1u;
    if (kept) {
      const __half2 X = __float2half2_rn(x.x), Y = __float2half2_rn(x.y), Z = __float2half2_rn(x.z);
      unsigned r[4];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const __half2 dx = __hmax2(__hsub2(__habs2(__hsub2(X, C[q][0])), H[q][0]), zero);
        const __half2 dy = __hmax2(__hsub2(__habs2(__hsub2(Y, C[q][1])), H[q][1]), zero);
        const __half2 dz = __hmax2(__hsub2(__habs2(__hsub2(Z, C[q][2])), H[q][2]), zero);
        const __half2 d2 = __hfma2(dz, dz, __hfma2(dy, dy, __hmul2(dx, dx)));
        const unsigned le = __hle2_mask(d2, rc2);
        r[2 * q] = __ballot_sync(0xffffffffu, keep && (le & 1u));
        r[2 * q + 1] = __ballot_sync(0xffffffffu, keep && (le >> 31));
      }
      I.r = make_uint4(r[0], r[1], r[2], r[3]);
      mycnt += __popc(cull_lanes(mine, I.r, kept));
    }
    if (lane == 0) {
      info[t].r = I.r;
      *reinterpret_cast<uint2*>(&info[t].kept) = make_uint2(I.kept, I.rest);
    }
  }
  if (lane < kCullClasses) cnt[wid][lane] = mycnt;
  else if (lane == kCullClasses) cnt[wid][lane] = rest;
  __syncthreads();
  // lane c: entries before class c, and before this warp's of class c; lane 16: the
  // tiles that stay tiles in the warps before
  int mycls = 0, before = 0;
  if (lane <= kCullClasses) {
#pragma unroll
    for (int w = 0; w < W; w++) {
      const int x = cnt[w][lane];
      mycls += x;
      before += w < wid ? x : 0;
    }
  }
  const int nrest = __shfl_sync(0xffffffffu, mycls, kCullClasses);
  int inc = lane < kCullClasses ? mycls : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  const int total = __shfl_sync(0xffffffffu, inc, 31);
  int off = (lane < kCullClasses ? inc - mycls : 0) + before;
  const int G = (total + 63) / 64 * 2;
  if (threadIdx.x == 0) {
    first_rest = nrest ? atomicAdd(&v.cull_n[0], nrest) : 0;
    first = G ? atomicAdd(&v.cull_n[1], G) : 0;
    if ((long long)(first + G) * 32 > v.cull_cap) v.cull_n[2] = 0;   // they do not fit: the tile path serves all
  }
  __syncthreads();
  const long long base = (long long)first * 32;
  if (base + (long long)G * 32 > v.cull_cap) return;
  for (int g = threadIdx.x; g < G; g += W * 32) v.cull_bi[first + g] = b;
  for (int i = total + threadIdx.x; i < G * 32; i += W * 32)
    v.cull_ent[base + i] = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
  const unsigned lt = (1u << lane) - 1u;
  int at_rest = first_rest + __shfl_sync(0xffffffffu, off, kCullClasses);
#pragma unroll 2
  for (int t = ta; t < tb; t++) {
    const uint2 k = *reinterpret_cast<const uint2*>(&info[t].kept);
    const unsigned kept = k.x;
    if (k.y && lane == 0) v.cull_rest[at_rest] = t;
    at_rest += k.y;
    if (!kept) continue;
    const uint4 r = info[t].r;
    const Tile T = v.tiles[t];
    const unsigned code = ((r.x >> lane) & 1u) | ((r.y >> lane) & 1u) << 1 | ((r.z >> lane) & 1u) << 2 |
                          ((r.w >> lane) & 1u) << 3;
    const int at = __shfl_sync(0xffffffffu, off, cull_class(code)) + __popc(cull_lanes(code, r, kept) & lt);
    if ((kept >> lane) & 1u) v.cull_ent[base + at] = make_float4(T.ox, T.oy, T.oz, __int_as_float(T.bj * 32 + lane));
    off += lane < kCullClasses ? __popc(cull_lanes(mine, r, kept)) : 0;
  }
}

static inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// grid of the warp-per-tile list kernels (grid-stride; 16 CTAs of 8 warps per SM)
static int list_tile_grid(const Context& c) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
  const long long want = (c.tile_cap + 7) / 8, g = 16LL * (sms > 0 ? sms : 1);
  return (int)(want < g ? (want > 0 ? want : 1) : g);
}

// exclusive scan of n ints (n <= 2^20): one CTA up to kScanOne, else two phases
static void scan_ints(Context& c, const int* in, int* out, int* tmp, long long n, cudaStream_t st) {
  c.kernel_launches += n <= kScanOne ? 1 : 2;
  if (n <= kScanOne) {
    launch_pdl(st, 1, 1024, 0, k_scan_one, in, out, (int)n);
    return;
  }
  const int nb = nblk(n, 1024);
  launch_pdl(st, nb, 1024, 0, k_scan_block, in, out, tmp, (int)n);
  launch_pdl(st, nb, 1024, 0, k_scan_add, out, tmp, (int)n);
}

// Whether some system may have its pairs in groups (the pair passes take them where they
// replace half of the tiles).  In a periodic box a tile stays a tile, with an image per
// pair, unless its blocks lie within L - R less their half-extents (some 5 A each in dense
// solvent) along every axis of edge L.  Water at R = 14 A, where half of the block pairs do
// from L = 39.7 A on: up to L = 38.3 no pass takes the groups, and building them costs 5
// to 12 us (L 27 to 38); at L = 42.1 they cost 15 us a build and take 10 us off each force
// pass, at 53.8 16 and 31.
static bool groups_serve(const Context& c, float R) {
  for (const SystemInfo& S : c.sys) {
    double f = 1.0;
    for (int k = 0; k < 3 && S.periodic; k++) f *= std::min(1.0, std::max(0.0, 2.0 * (S.box[k] - R - 10.0) / S.box[k]));
    if (f >= 0.5) return true;
  }
  return false;
}

// NB j-atom groups: only where the per-step displacement check runs
static bool makes_groups(const Context& c, float list_radius) {
  return c.nb_set && c.nb_cull && c.lp.check_skin && c.cull_cap > 0 && groups_serve(c, list_radius);
}

static void launch_cull(Context& c, float list_radius) {
  c.kernel_launches += 1;
  const float R = list_radius + 1e-3f, Rc = fmaxf(list_radius - (float)c.lp.Padding, 0.f);
  CullTile* info = reinterpret_cast<CullTile*>(c.d_cull_mask.p);
  if (c.nblocks <= 8 * 152)
    launch_pdl(c.stream, c.nblocks, 16 * 32, 0, k_cull<16>, c.view(), R * R, Rc * Rc, c.d_row_start.p, c.d_row_cnt.p, info);
  else
    launch_pdl(c.stream, c.nblocks, 8 * 32, 0, k_cull<8>, c.view(), R * R, Rc * Rc, c.d_row_start.p, c.d_row_cnt.p, info);
}

// the overflow flag of a build about to be repeated into grown arrays
__global__ void k_clear_status(unsigned* status, unsigned bits) { atomicAnd(status, ~bits); }
static int clear_tile_overflow(Context& c) {
  c.kernel_launches += 1;
  k_clear_status<<<1, 1, 0, c.stream>>>(c.d_status.p, (unsigned)ST_TILE_OVERFLOW);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

static void launch_rows(Context& c, float R, float full_radius) {
  const int words = (c.max_sys_blocks + 31) / 32 + 1;
  const size_t smem = (size_t)2 * words * sizeof(unsigned);
  int* cnt = c.d_counters.p;
  launch_pdl(c.stream, c.nblocks, kRowWarps * 32, smem, k_tile_rows, c.view(), c.d_bgrid.p, reinterpret_cast<int*>(c.d_sys_hmax.p), c.d_bcell_off.p, c.d_bcell_count.p,
      c.d_bcell_blocks.p, c.d_slot_of.p, R, (float)c.lp.Padding, full_radius, c.full_margin(), c.d_row_cnt.p,
      c.d_row_start.p, c.tile_cap, words, cnt + 6, c.d_mlist.p, cnt + 7);
}

static SlotParams slot_param_view(const Context& c) {
  SlotParams P;
  P.radius = c.d_radius.p;
  P.sqeps = c.d_sqeps.p;
  P.gbR = c.has_gb ? c.d_gbR.p : nullptr;
  P.gbVj = c.has_gb ? c.d_gbVj.p : nullptr;
  P.lcR = c.has_sa ? c.d_lcpoR.p : nullptr;
  P.lcUse = c.has_sa ? c.d_lcpoUse.p : nullptr;
  P.lc_par = c.has_sa ? c.d_lc_par.p : nullptr;
  P.charge = c.d_charge.p;
  return P;
}

// the part of a build after its rows: masks, GB work items, NB groups
static void launch_list_tail(Context& c, float list_radius) {
  cudaStream_t st = c.stream;
  int* cnt = c.d_counters.p;
  c.kernel_launches += 1;
  const int gm = nblk((long long)c.mask_cap * 32, 256), gt = list_tile_grid(c);
  launch_pdl(st, gm < gt ? gm : gt, 256, 0, k_masks, c.view(), c.d_slot_of.p, c.d_mlist.p, cnt + 7, cnt + 6, c.tile_cap);
  if (c.has_gb) {
    c.kernel_launches += 1;
    const int far = c.gb_set && make_gb_const(c.gb, list_radius).far_inner > 0.f ? 1 : 0;
    launch_pdl(st, nblk(c.nblocks, 4), 128, 0, k_items, c.view(), c.gb_item_tiles == 2 ? 1 : 0, far, c.d_row_start.p,
                                                c.d_row_cnt.p);
  }
  c.cull_built = makes_groups(c, list_radius);
  if (c.cull_built) launch_cull(c, list_radius);
}

static ListState list_state(Context& c, bool grid, bool groups) {
  ListState I;
  I.count = c.d_count.p;
  I.head = c.d_head.p;
  I.lo = reinterpret_cast<int*>(c.d_sys_lo.p);
  I.hi = reinterpret_cast<int*>(c.d_sys_hi.p);
  I.hmax = reinterpret_cast<int*>(c.d_sys_hmax.p);
  I.bcell_count = c.d_bcell_count.p;
  I.bcell_cursor = c.d_bcell_cursor.p;
  I.counters = c.d_counters.p;
  I.ncells = c.nsys * kCellsPerSystem;
  I.nbcells = grid ? c.nblocks : 0;
  I.nsys3 = 3 * c.nsys;
  I.groups = groups ? 1 : 0;
  return I;
}

// (once, before a context's first build)
int launch_list_init(Context& c) {
  k_list_init<<<std::min(nblk(std::max(c.nsys * kCellsPerSystem, c.nslots), 256), 1216), 256, 0, c.stream>>>(
      list_state(c, false, false), c.d_sorted_atom.p, c.nslots);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

int launch_list_build(Context& c, float list_radius, float full_radius, ListSizing sizing) {
  c.kernel_launches += 4;
  DevView v = c.view();
  cudaStream_t st = c.stream;
  const bool grid = c.max_sys_blocks > kDirectBlocks;
  ListState I = list_state(c, grid, makes_groups(c, list_radius));
  if (!c.all_periodic) {
    c.kernel_launches += 1;
    launch_pdl(st, nblk(c.natom, 256), 256, 0, k_bbox, v, c.d_atom_sys.p, I.lo, I.hi);
  }
  const Spread ks = spread(c.natom, 64);
  launch_pdl(st, ks.grid + (grid ? 1 : 0), ks.threads, 0, k_keys, v, c.d_atom_sys.p, I, c.d_next.p, c.d_cell.p,
             grid ? c.d_bgrid.p : nullptr);
  launch_pdl(st, nblk(I.ncells, 1024), 1024, 0, k_scan_block, c.d_count.p, c.d_offset.p, c.d_scan_tmp.p, I.ncells);
  launch_pdl(st, nblk(I.ncells, kSortThreads), kSortThreads, 0, k_cell_sort, v, I, c.d_offset.p, c.d_scan_tmp.p, c.d_next.p,
             c.d_cell.p, c.d_tmp_sorted.p, c.d_sorted_atom.p, c.d_slot_of.p);
  launch_pdl(st, nblk((long long)c.nblocks * 32, 128), 128, 0, k_blocks, v, slot_param_view(c), c.clear, c.d_bgrid.p, I.hmax, c.d_bcell.p,
                                                                 c.d_bcell_count.p, c.nb_set ? 1 : 0);
  if (grid) {
    c.kernel_launches += 1;   // and a scan
    scan_ints(c, c.d_bcell_count.p, c.d_bcell_off.p, c.d_bcell_scan_tmp.p, c.nblocks, st);
    launch_pdl(st, nblk(c.nblocks, 256), 256, 0, k_bgrid_scatter, v, c.d_bcell.p, c.d_bcell_off.p, c.d_bcell_cursor.p,
                                                           c.d_bcell_blocks.p);
  }
  launch_rows(c, list_radius, full_radius);
  if (sizing != kListDevice) {
    // the tile count against the capacity: a list that outgrew the arrays is
    // rebuilt into grown ones.  The rest of the build is queued behind the copy of
    // the count, so the GPU works on while the host waits for it (a list that did
    // not fit is cut to the capacity, and the rest runs again after the growth)
    if (cudaMemcpyAsync(c.h_total.p, c.d_counters.p + 6, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaEventRecord(c.ev_total, st) != cudaSuccess)
      return PDGPU_ERR_CUDA;
    if (c.tile_cap > 0) launch_list_tail(c, list_radius);
    if (cudaEventSynchronize(c.ev_total) != cudaSuccess) return PDGPU_ERR_CUDA;
    const int total = *c.h_total.p;
    if (total > c.tile_cap) {
      // (the overflow of the arrays just outgrown is no error of this build)
      if (clear_tile_overflow(c) != PDGPU_OK) return PDGPU_ERR_CUDA;
      if (sizing == kListCheck) return PDGPU_ERR_CAPACITY;
      if (cudaStreamSynchronize(st) != cudaSuccess) return PDGPU_ERR_CUDA;
      const int e = alloc_tiles(c, total);
      if (e != PDGPU_OK) return e;
      c.kernel_launches += 1;
      I.groups = makes_groups(c, list_radius) ? 1 : 0;
      launch_pdl(st, 1, 32, 0, k_reset_counters, I);
      launch_rows(c, list_radius, full_radius);
      launch_list_tail(c, list_radius);
    }
  } else {
    launch_list_tail(c, list_radius);
  }
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

int launch_slot_params(Context& c) {
  c.kernel_launches += 1;
  k_slot_params<<<nblk(c.nslots, 256), 256, 0, c.stream>>>(c.view(), slot_param_view(c));
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

PackArgs pack_args(const Context& c, float check_disp) {
  PackArgs P{};
  P.charge = c.d_charge.p;
  P.clear = c.clear;
  P.check2 = check_disp > 0 ? check_disp * check_disp : 0.f;
  if (c.full_radius_built > 0.f) {
    const float h = 0.5f * c.full_margin();
    P.full2 = h * h;
  }
  P.npairs_all = c.npairs_all;
  P.cull = c.cull_built ? 1 : 0;
  P.gb = c.has_gb ? 1 : 0;
  return P;
}

int launch_pack(Context& c, float check_disp) {
  c.kernel_launches += 1;
  const Spread sp = spread(c.nslots, 64);   // (32: 1 us a step slower at 2,001 atoms)
  launch_pdl(c.stream, sp.grid, sp.threads, 0, k_pack, c.view(), pack_args(c, check_disp));
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

}  // namespace pdgpu
