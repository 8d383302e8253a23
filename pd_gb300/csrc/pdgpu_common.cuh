// pdgpu_common.cuh — shared definitions for the GB300 nonbonded / GB / LCPO path.
//
// Layout (one context may hold several independent systems, "a batch"):
//   * original order  : atoms as the host numbers them, systems concatenated.
//   * sorted order    : per system, atoms ordered along a 3-D Hilbert curve of a
//                       32^3 cell grid, padded to a multiple of 32; slot s holds
//                       original atom sorted_atom[s] (or -1 for padding).
//   * blocks          : 32 consecutive sorted slots of one system.
//   * tiles           : block pairs (bi <= bj) of one system whose bounding boxes
//                       come within the list radius; one warp evaluates the
//                       32x32 interactions of a tile by shuffle rotation.
// Forces, Born-radius sums, dE/da and energies are accumulated in 64-bit fixed
// point, so results are bit-identical run to run whatever the tile order.
// Internal units: Angstrom, kcal/mol, e; conversion to PD units (J, N) happens
// once per atom / per energy at the end.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/pdgpu.h"
#include "pdgpu_df.cuh"

namespace pdgpu {

constexpr int kWarp = 32;
constexpr int kHilbertBits = 5;                       // 32 cells per dimension
constexpr int kCellsPerSystem = 1 << (3 * kHilbertBits);
constexpr int kMaxSystemBlocks = 65536;               // blocks of one system (2^21 atoms): the list-build bitmap
constexpr int kBandWidth = 64;                        // bonded partners within +-64 indices use the band masks
constexpr int kLcpoMax = 80;                          // PD caps an atom's LCPO overlap list at 80 (lcpo.h:24)
constexpr int kLcpoCand = 160;                        // candidate capacity before the cap is applied

// fixed-point scales
constexpr double kForceScale = 4294967296.0;          // 2^32 per kcal/mol/A
constexpr double kEnergyScale = 4294967296.0;         // 2^32 per kcal/mol (|E| < 2^31 kcal/mol per slot)
constexpr double kSumScale = 4294967296.0;            // 2^32 per unit (Born sums, dE/da)

// per-system energy slots (fixed point)
enum EnergySlot { E_VDW = 0, E_ELEC, E_POL_CROSS, E_POL_SELF, E_SURF, E_VIRIAL, E_BOND, E_ANGLE, E_TORS, E_IMPR, E_NSLOTS };

// status bits set by kernels
enum StatusBits : unsigned {
  ST_LCPO_OVERFLOW = 1u,
  ST_FIXED_OVERFLOW = 2u,
  ST_NAN = 4u,
  ST_STALE_LIST = 8u,
  // the tile list or its exclusion-mask table outgrew its capacity in a build
  // that could not resize it (a captured step); the list is incomplete
  ST_TILE_OVERFLOW = 16u,
};

struct SystemInfo {
  int atom_start;   // first atom (original order)
  int natom;
  int pad_start;    // first slot (sorted order)
  int npad;         // multiple of 32
  int block_start;
  int nblocks;
  int grid_start;   // first cell of this system's block grid (list build)
  int grid_cells;   // its cell budget: one per block
  int periodic;
  double box[3];
  double ibox[3];   // 1 / box (periodic systems)
  DF boxf[3];       // box as double-floats
  float boxt[3];    // and what these leave of it
};

struct __align__(16) Tile {
  int bi, bj;
  int mask;    // index into the exclusion-mask table or -1
  int flags;   // bit0: per-pair minimum image needed, bit1: diagonal tile,
               // bit2: every pair inside all cutoffs and switch radii (with margin)
  // centre of block bj seen from block bi (its periodic image in a box), formed
  // in FP64 at the list build and rounded once: the pair kernels add it to the
  // j positions without per-tile FP64 work
  float ox, oy, oz, pad;
};

// Grid over one system's block centres (list build), remade every build: cells
// of about equal edge over the periodic box, or over the bounding box of the
// system's atoms in open space, at most one cell per block
struct BlockGrid {
  double origin[3];
  double cell[3];   // cell edges
  int dims[3];
  int start;        // first cell in the context's cell arrays
};

// Pair-law constants for the LJ + Coulomb kernel (FF_NonBonded)
// (the _d members are the same constants in FP64, for the energy arithmetic)
struct NBConst {
  float cut2, vdwcut2, vdw14, elec14, econv_diel;
  double cut2_dd, vdwcut_d, vdwinner_d, inner_d, vdwinvw2_d, invw2_d, econv_diel_d, vdw14_d, elec14_d;
  double sA, sB, sC, sD, sE, fsw_cutV, eshift, cut2_d, inner2_d;
  // FP32 copies for the force pair law
  float vdwcut_f, vdwinner_f, vdwinvw2_f, inner_f, invw2_f, inner2_f, sA_f, fsw_k;  // fsw_k = cut2 - 3 inner2
  int elecmode;            // 0 none, 1 plain, 3 energy switch, 4 force switch
  int dovdw;
  // 1: LJ and Coulomb switched over the same radii (Cutoff = VdwCutoff,
  // InnerCutoff = VdwInnerCutoff, energy switch, LJ on): one switch serves both
  int samesw;
  // 1: LJ and Coulomb (if any) both end by a switch, LJ not beyond Cutoff, so the
  // law is continuous at every cutoff (the packed force pass)
  int smooth;
};

// The same constants as double-floats, for the pair energies (FF_NonBonded)
struct NBEConst {
  DF econv, vdw14, elec14;
  DF vdwcut, vdwinner, vdwinvw2, inner, invw2;
  DF sA, eshift, cut, cut2, fsw_k;                    // fsw_k = cut2 - 3 inner2
  // the force switch's energy is qq sA (C - r)^3 Q(r) / r with Q = q0 + q1 r + q2 r^2 + q3 r^3:
  // PD's sum of powers and its value at C, of which little is left at r near C, divided by
  // their triple root
  DF q0, q1, q2, q3;
  float vdwinner_t, inner_t, cut_t, cut2_t, fsw_t, eshift_t;   // what the double-floats leave of these
  int dovdw, vdw_hard;   // vdw_hard: LJ ends at VdwCutoff without a switch
};

// Constants for the GB fast path (FF_GeneralizedBorn_Still::calcForcesIncludingVacuo)
struct GBConst {
  float cut2, inner, invw2, vdwcut, vdwinner, vdwinvw2;
  float still2;            // min(GbsaStillCutoff, list radius)^2
  float econv_in, econv_out, premul;  // kcal units
  float vdw14, elec14, thresh;
  float P4, P5, invP5;
  float born2;             // the power of two next to P4: what the Born sums carry of it
  double still2_d, thresh_d;
  // 1: FastMode (GB fused with LJ + Coulomb, eps_out Coulomb below the threshold);
  // 0: calcBornForces (GB term alone for every pair, premul q q / r below it)
  int fast;
  // energy passes: pairs closer than sqrt(eclose2) take their energies in
  // double-float from double-float positions and parameters
  float eclose2;
  DF econv_in_f, econv_out_f, premul2_f, vdw14_f, elec14_f, eout_f;   // premul2: 2 premul
  // the packed pair bodies: a_i a_j K >= r^2 holds for every pair the threshold test
  // may switch on (K = -4 x the threshold widened by 4e-6 relative); force-only passes
  // scale the Born radii by sqrtK.  Tile pairs scale charges by sqrt(econv_out) (the
  // held atoms' by its negative) and sqrt(eps) by sqrt(12); single tiles, which hold
  // the close pairs, take the atoms' values as they are (eout = econv_out).  gb_ep: premul q q fgb per -econv_out q q
  // far_inner: the smallest inner cutoff where it is 64 A or more (0 otherwise):
  // tiles inside it are worth finding by their blocks' radii (tile_full_now)
  float far_inner;
  float K, sqrtK, inv_sqrtK, invK, kU, sq_eout, neg_sq_eout, eout, in_over_out, sqrt12, gb_ep;
};

// Where component c of slot s lies in a force accumulator: a block's 32 x sums, its y
// sums, its z sums.  A warp adds one component of consecutive slots with one
// instruction; 8 bytes apart they fill 8 sectors, 24 bytes apart they touch 24.
__host__ __device__ __forceinline__ size_t force_at(int s, int c) { return (size_t)(s >> 5) * 96 + 32 * c + (s & 31); }

// Device-side view of a context, passed by value to kernels.
struct DevView {
  int nsys, natom, nslots, nblocks;
  const SystemInfo* sys;
  const int* slot_sys;       // [nblocks] system of each block
  // original order
  const double* pos;         // natom*3
  const double* charge;      // natom, e
  const double* radius;      // natom, LJ Rmin/2
  const double* sqeps;       // natom, sqrt(kcal/mol)
  const double* born;        // natom, Born radii of the last GB pass (FP64)
  // sorted order
  const int* sorted_atom;    // [nslots]
  float4* xq;                // rel pos + charge
  float4* par;               // LJ radius, sqrt(eps kcal), GB R (raw), GB Vj
  float4* rel0;              // rel pos at list build (displacement check)
  double* center;            // [nblocks*3]
  float4* half;              // [nblocks] half extents
  float4* sub;               // [nblocks*8] box (lo, hi) of each 8 slots at the packed positions, in the block's frame
  float* brad;               // [nblocks] (GB) radius about the centre at the packed positions, rounded up
  const float* bborn;        // [nblocks] largest Born radius of the last GB pass
  float4* cenf;              // [nblocks] centre in FP32 (exact: centres are FP32 numbers)
  // (energy evaluations) what FP32 rounding takes off the packed slots:
  // (x, y, z, charge) - xq and (LJ radius, sqrt(eps)) - par, written before the energy pass
  float4* rlo;
  float2* plo;
  unsigned long long* band_excl;   // per atom: bit d-1 => partner i+d excluded (bo<=2)
  unsigned long long* band_14;     // per atom: bit d-1 => partner i+d is a 1-4 pair
  const unsigned long long* band_dn_excl;   // the same for partners of lower index: bit d-1 => i-d
  const unsigned long long* band_dn_14;
  const int* far_both_start; // CSR of the bonded partners beyond the band, of either side
  const int* far_both_idx;
  const int* far_both_bo;
  const int* far_start;      // CSR of partners beyond the band, per atom
  const int* far_idx;
  const int* far_bo;
  Tile* tiles;
  int* ntiles;
  // GB work items over the tile list: a pair of all-inside tiles of one row
  // (x, y), or a single tile (x, -1)
  int2* items;
  int* nitems;
  uint2* masks;              // [mask_cap*32] per lane: (excluded bits, 1-4 bits) in rotation order
  int* nmasks;
  int mask_cap;
  // NB j-atom groups: per i-block row, the j atoms of its unmasked, off-diagonal,
  // single-image tiles that lie within the list radius of the i block's box,
  // packed 32 to a group; the other tiles stay on the tile path (cull_rest)
  float4* cull_ent;          // [cull_cap] j offset into the i block's frame (x, y, z), j slot (int bits; -1 empty)
  int* cull_bi;              // [cull_cap / 32] i block of each group (a row's groups: an even number)
  int* cull_rest;            // [tile capacity] tiles left on the tile path (any order)
  int* cull_n;               // [0] rest tiles, [1] groups, [2] 1 when the groups fit the capacity
  long long cull_cap;        // entries
  long long* facc;           // [nslots*3], component c of slot s at force_at(s, c)
  long long* eacc;           // [nsys*E_NSLOTS]
  unsigned* status;
};

// What an evaluation clears before it accumulates: the pass that packs the
// positions does it (null pointers are skipped), so a step launches no memsets
struct StepClear {
  long long *facc, *gpol, *deda;     // per slot (facc: 3)
  long long *facc2;                  // per slot, 3: the cached LCPO forces before their recalculation
  long long *eacc, *surf, *ke;       // per system (eacc: E_NSLOTS)
};
__device__ __forceinline__ void step_clear(const StepClear& C, const DevView& v, int s) {
  if (C.facc) C.facc[force_at(s, 0)] = C.facc[force_at(s, 1)] = C.facc[force_at(s, 2)] = 0;
  if (C.gpol) C.gpol[s] = 0;
  if (C.deda) C.deda[s] = 0;
  if (C.facc2) C.facc2[force_at(s, 0)] = C.facc2[force_at(s, 1)] = C.facc2[force_at(s, 2)] = 0;
  if (C.eacc)   // (no fewer slots than 32 per system: every entry of a system's has a slot)
    if ((s & 31) < E_NSLOTS && s == 32 * v.sys[v.slot_sys[s >> 5]].block_start + (s & 31))
      C.eacc[(size_t)v.slot_sys[s >> 5] * E_NSLOTS + (s & 31)] = 0;
  if ((C.surf || C.ke) && s == 32 * v.sys[v.slot_sys[s >> 5]].block_start) {
    if (C.surf) C.surf[v.slot_sys[s >> 5]] = 0;
    if (C.ke) C.ke[v.slot_sys[s >> 5]] = 0;
  }
}

// Programmatic dependent launch.  A kernel launched with launch_pdl may be put on
// the SMs as soon as every CTA of its predecessor in the stream has started;
// pdl_sync, the first thing it does, lets its own successor do the same and then
// waits until the predecessor has finished and its writes are visible.  Every
// kernel of the evaluation's main chain does both, so the order of the chain
// holds across any number of kernels, and the launch latency between two of them
// (~2 us, ten of them in a small system's step) is hidden.
__device__ __forceinline__ void pdl_sync() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(cudaStream_t st, unsigned grid, unsigned block, size_t smem, void (*kernel)(P...), A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ---------------------------------------------------------------------------
// fixed point helpers
// ---------------------------------------------------------------------------
// energies: 2^32 per kcal/mol.  The resolution matters: a converted partial
// sum keeps only whole units, so many small partial sums of one sign (the far
// attractive LJ tail, per lane and tile) would be lost at a coarse scale.
__device__ __forceinline__ long long fix_energy_d(double x) { return __double2ll_rn(x * 4294967296.0); }
// float -> 64-bit fixed point with 32 fractional bits (|x| < 2^29; fix_range flags
// anything from 2^28 on): x = a / 4 + rem with a the nearest integer to 4 x, both
// exact in FP32, so x 2^32 = a 2^30 + rem 2^32 takes three 32-bit conversions.
// Rounds to nearest even (exact ties, common where x is small, do not drift one
// way).  The hardware float -> int64 conversion runs on the narrow FP64 pipe, and
// shifting the mantissa by the exponent in integers takes about twenty instructions.
__device__ __forceinline__ long long fx32(float x) {
  const int a = __float2int_rn(x * 4.f);
  const float rem = __fmaf_rn(-(float)a, 0.25f, x);
  return (long long)a * 1073741824LL + (long long)__float2int_rn(rem * 4294967296.f);
}

// the status code of a set of status bits
inline int status_code(unsigned st) {
  if (st & ST_NAN) return PDGPU_ERR_NAN;
  if (st & ST_FIXED_OVERFLOW) return PDGPU_ERR_FIXED_OVERFLOW;
  if (st & (ST_LCPO_OVERFLOW | ST_TILE_OVERFLOW)) return PDGPU_ERR_LIST_OVERFLOW;
  if (st & ST_STALE_LIST) return PDGPU_ERR_STALE_LIST;
  return PDGPU_OK;
}

// Range of FP32 partial sums about to enter 64-bit fixed point (2^32 per unit):
// m is the sum of their magnitudes.  NaN or infinity sets ST_NAN; 2^28 or more
// sets ST_FIXED_OVERFLOW.  One conversion holds up to 2^30 and a slot's total
// up to 2^31, so flagging every partial sum at 2^28 keeps a few large ones
// from wrapping a total past the final check unnoticed.  (PD has no such
// limit; 2^28 kcal/mol/A lies far beyond any physical force.)
__device__ __forceinline__ void fix_range(unsigned* status, float m) {
  if (!(m < 268435456.f)) atomicOr(status, !(m < 1.0e18f) ? (unsigned)ST_NAN : (unsigned)ST_FIXED_OVERFLOW);
}

__device__ __forceinline__ void atomic_add_ll(long long* p, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(v));
}
__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// host-side launchers (defined in the .cu files)
// ---------------------------------------------------------------------------
struct Context;
int tile_grid(Context& c);   // grid of the tile kernels (grid-stride, one tile per warp item)
// full_radius: distance below which every cutoff and switch of the set
// components is inactive (0 = never mark tiles full).  sizing: how the tile
// count meets the capacity:
//   kListReadback  read the count back, grow the tile arrays when it exceeds them
//   kListCheck     read it back, PDGPU_ERR_CAPACITY when it exceeds them (no allocation)
//   kListDevice    no host round trip (a captured step): an overflow leaves the
//                  list short and sets ST_TILE_OVERFLOW
enum ListSizing { kListReadback = 0, kListCheck = 1, kListDevice = 2 };
int launch_list_build(Context& c, float list_radius, float full_radius, ListSizing sizing);
// tile arrays (and the NB group arrays sized from them) for `tiles` tiles
int alloc_tiles(Context& c, long long tiles);
// the NB j-atom group arrays for the current tile capacity
int alloc_cull_tiles(Context& c);
int launch_list_init(Context& c);
int launch_pack(Context& c, float check_disp);
int launch_nb(Context& c, const NBConst& k, bool energy, bool forces);
int launch_gb(Context& c, const GBConst& k, double halfeconv, double born_offset, double premul, bool energy);
int launch_lcpo(Context& c, long long* facc_out, long long* esurf_out, int esurf_stride);
// FP32 remainders of the packed slots (double-float positions and parameters), before an energy pass
int launch_df_records(Context& c);
int launch_gb_stage(Context& c, const GBConst& k, int stage);
// parameter gradients (device outputs, original atom order, J per parameter unit;
// null pointers are skipped): scratch, cleared, filled by the energy pass of NB or
// GB (GB: the pair terms' gradients, launch_adj_gb_pair) and finished here
struct AdjScratch {
  long long* g = nullptr;   // fixed-point sums, 5 per slot
  float* w = nullptr;       // dE/dGpol per slot
};
int adjoint_scratch(Context& c, AdjScratch& a);
// a static device array: no allocation during the call (at most kNoAllocMaxSlots
// sorted slots; one scratch per device shared by all contexts)
constexpr int kNoAllocMaxSlots = 65536;
int adjoint_scratch_static(Context& c, AdjScratch& a);
int clear_adjoint(Context& c, const AdjScratch& a);
int launch_adj_gb_pair(Context& c, const GBConst& k);
int launch_adjoint(Context& c, unsigned what, const AdjScratch& a, double* d_q, double* d_r, double* d_e, double* d_R,
                   double* d_V, double* d_T);
// Monte Carlo partial NB energies: take the reference from the last energy
// evaluation / update it by the pairs of the moved atoms
int launch_mc_reference(Context& c);
int launch_mc_update(Context& c);
// static per-slot parameters refreshed from the per-atom arrays (after a parameter update)
int launch_slot_params(Context& c);
// measurement aids (k_diag.cu): the pair census of the current list into out[5]
// (device, zeroed by the caller) and the FP32 FMA ceiling of a device
int launch_census(Context& c, const NBConst& nk, const GBConst& gk, bool do_nb, bool do_gb, unsigned long long* out);
int measure_fp32_peak(int device, double* tflops_ffma, double* tflops_ffma2);
NBConst make_nb_const(const pdgpu_nb_params& p);
NBEConst make_nbe_const(const NBConst& k);
double born_sum_unit(const pdgpu_gb_params& p);     // Gpol per unit of the Born sums' fixed point
void set_gb_threshold(GBConst& k, double thresh);   // ExpApproxThreshold and what the bodies derive from it
GBConst make_gb_const(const pdgpu_gb_params& p, double listR);
int launch_bonded(Context& c, bool energy);
int launch_finalize_forces(Context& c, double* out, size_t stride_doubles, bool add, double scale);
// host-side orchestration shared by the evaluation and dynamics entry points
int rebuild_list_impl(Context& c);
void release_streams(Context& c);
int enqueue_forces(Context& c, unsigned what, bool energy, bool rebuild, long long* lcpo_f, long long* lcpo_e,
                   int lcpo_e_stride, bool run_lcpo, bool packed = false);
struct MDState;
void destroy_md(Context& c);
// captured step graphs hold buffer addresses: dropped when a buffer is replaced
void drop_step_graphs(Context& c);

}  // namespace pdgpu
