// k_gb.cu — Still Generalised Born (FastMode).
//
// PD src/mmlib/forcefields/gbff.cpp:
//   Born radii            calcBornRadii_PairwiseApprox   :432-483
//   fused GB+LJ+Coulomb   calcForcesIncludingVacuo loop1 :1546-1746 (+ self term :1740-1745)
//   Born-radius chain     calcForcesIncludingVacuo loop2 :1768-1825
// GB uses plain Euclidean distances, as PD does.
//
// Work decomposition: one warp per GB work item (grid-stride over the item list
// the list build writes): a tile pair (bi, bj), (bi, bj + 1) of one row whose
// pairs all lie inside every cutoff, or single 32x32 tiles.  In a tile pair each
// lane holds one atom of each j block and the shared bi block rotates, so one
// rotation serves two pairs.  A single tile (masked, diagonal, odd, or cut by a
// cutoff) is step-packed: lane l holds i atom l and takes the j atoms l + kk and
// l + kk + 1 of the rotating block as one FP32x2 pair, read from the warp's rows
// in shared memory; its exclusion bits are tested per half.  Both run on packed
// f32x2 arithmetic.  Every FP32 sum is converted to 64-bit fixed point and added
// atomically once per tile (so a slot's total does not depend on the order in
// which items run).  Registers decide the occupancy of these kernels.
#include "pdgpu_tile.cuh"

namespace pdgpu {

// ---------------------------------------------------------------------------
// pass 1: Born-radius pair sums  Gpol_i += P4 Vj CCF / r^4  (bond order > 2).  The sums
// carry the power of two next to P4 (GBConst::born2, exact in every volume); the rest of
// P4 meets them in FP64 (k_gb_radii): rounded with P4 in it, a volume would shift the sums
// of all its partners alike.
// ---------------------------------------------------------------------------
// inside GbsaStillCutoff (FULL: the whole tile is); pairs within FP32 rounding of
// the cutoff are decided in FP64
template <bool FULL>
__device__ __forceinline__ bool still_in(const DevView& v, const GBConst& k, float r2, int sa, int sb) {
  if (FULL) return true;
  bool in = r2 <= k.still2;
  if (fabsf(r2 - k.still2) <= 2e-6f * k.still2) in = r2_slots_fp64(v, sa, sb) <= k.still2_d;
  return in;
}

// Close contact, r^2 / (R_i + R_j)^2 <= 1 / P5, where the CCF switches on.  Tested
// as r^2 <= rs^2 / P5 (no division); the CCF is continuous there (h = 1), so
// the rounding of the test does not matter.  Rare in a tile: the bodies take
// the branch only when some lane of the warp needs it (a warp vote), so the
// trigonometric code is skipped, not predicated, on nearly every step.
__device__ __forceinline__ bool gb_contact(const GBConst& k, float r2, float rs2) { return r2 <= rs2 * k.invP5; }

// ---------------------------------------------------------------------------
// All-inside tile pairs (every pair inside every cutoff, no exclusions: the
// all-pairs case) take lean Born and chain-rule bodies: per-atom factors are
// folded into the values loaded once per item, and the close-contact (CCF)
// branch is entered on a warp vote over a coarse bound of the item,
// (max R_i + max R_j)^2 / P5, instead of each pair's own limit.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// Tile pairs far from their row's block skip a branch for the whole item: every
// pair of the item lies farther apart than sqrt(lim), lim a bound over the
// rotating block for each of the lane's two held atoms.  The rotating block sits
// at the origin of the item's frame, so a held atom at x keeps at least
// |x| - rho from it, rho the block's radius at the current positions.
__device__ __forceinline__ bool item_far(const float4& xa, const float4& xb, const float4& xr, float lima, float limb) {
  const float rho = sqrtf(warp_max(xr.x * xr.x + xr.y * xr.y + xr.z * xr.z));
  const float da = sqrtf(xa.x * xa.x + xa.y * xa.y + xa.z * xa.z) * 0.99999f - rho;
  const float db = sqrtf(xb.x * xb.x + xb.y * xb.y + xb.z * xb.z) * 0.99999f - rho;
  return __all_sync(0xffffffffu, da > 0.f && db > 0.f && da * da > lima && db * db > limb);
}

// an upper bound of (R_i + R_j)^2 / P5 over the pairs of a tile pair: held raw
// GB radii RS, the rotating block's Rr
__device__ __forceinline__ float pair_contact2(const GBConst& k, float2 RS, float Rr) {
  const float m = warp_max(fmaxf(RS.x, RS.y)) + warp_max(Rr);
  return m * m * k.invP5 * 1.0001f;
}

// Step-packed lean bodies (Born, chain rule): lane l takes the rotating
// block's atoms l + kk and l + kk + 1 as one FP32x2 register pair, so a packed
// instruction covers two rotation steps of one held atom, whose values are
// broadcast into both halves once per item.  The rotating block is staged once
// per item in the warp's own shared-memory rows as step pairs (x_l, x_l+1,
// y_l, y_l+1) ..., read with one 16-byte load per four values; only its running
// sums rotate through the warp by shuffles, two lanes per step, so that after
// 16 rotations lane l's pair holds the sums of atoms l and l + 1.
// the CCF of one pair: 1 outside close contact
__device__ __forceinline__ float born_ccf(const GBConst& k, float r2, float rs) {
  const float rs2 = rs * rs;
  if (!gb_contact(k, r2, rs2)) return 1.f;
  const float h = 0.5f - 0.5f * cospif(__fdividef(r2, rs2) * k.P5);
  return h * h;
}

constexpr int kBornThreads = 256;
constexpr int kBornWarps = kBornThreads / 32;

// rows of the rotating block in the warp's shared memory, twice over, so that a
// lane's row at step kk lies at a fixed offset from its first (no wrap-around)
struct BornRows {
  float4 xy[64], zv[64];   // (x, x', y, y'), (z, z', V, V'); with the base law (x, y, z, q), (LJ R, sqrt(12 eps), V, -) (V: times born2)
  float2 r[64];            // (R, R'), single tiles only
};

// Born sums of a single tile, step-packed (MASKED: exclusion bits and the
// diagonal; FULL: every pair inside the Still cutoff)
template <bool MASKED, bool FULL>
__device__ __forceinline__ void born_tile(const DevView& v, const GBConst& k, const Tile& T, int lane, unsigned ex,
                                          long long* gpol, BornRows& rs) {
  const int si = T.bi * 32 + lane, j0 = T.bj * 32, l1 = (lane + 1) & 31;
  const float4 xi = v.xq[si], pi = v.par[si];
  {
    const float4 x0 = j_in_i_frame(v, T, lane), p0 = v.par[j0 + lane];
    const float v0 = k.born2 * p0.w;
    const float x1 = __shfl_sync(0xffffffffu, x0.x, l1), y1 = __shfl_sync(0xffffffffu, x0.y, l1);
    const float z1 = __shfl_sync(0xffffffffu, x0.z, l1), v1 = __shfl_sync(0xffffffffu, v0, l1);
    const float r1 = __shfl_sync(0xffffffffu, p0.z, l1);
    __syncwarp();
    rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x1, x0.y, y1);
    rs.zv[lane] = rs.zv[lane + 32] = make_float4(x0.z, z1, v0, v1);
    rs.r[lane] = rs.r[lane + 32] = make_float2(p0.z, r1);
    __syncwarp();
  }
  const float2 AX = f2(-xi.x), AY = f2(-xi.y), AZ = f2(-xi.z), RA = f2(pi.z), VA = f2(k.born2 * pi.w);
  float2 GA = f2(0.f), GR = f2(0.f);
#pragma unroll 4
  for (int kk = 0; kk < 32; kk += 2) {
    const int j = lane + kk;
    const float4 P = rs.xy[j], Q = rs.zv[j];
    const float2 ax = __fadd2_rn(make_float2(P.x, P.y), AX), ay = __fadd2_rn(make_float2(P.z, P.w), AY);
    const float2 az = __fadd2_rn(make_float2(Q.x, Q.y), AZ);
    const float2 r2 = __ffma2_rn(az, az, __ffma2_rn(ay, ay, __fmul2_rn(ax, ax)));
    const float2 ir2 = make_float2(rcp_ftz(r2.x), rcp_ftz(r2.y));
    float2 w = __fmul2_rn(ir2, ir2);
    const float2 s = __fadd2_rn(rs.r[j], RA), s2 = __fmul2_rn(s, s), lim = __fmul2_rn(s2, f2(k.invP5));
    if (__any_sync(0xffffffffu, r2.x <= lim.x || r2.y <= lim.y)) {
      w.x *= born_ccf(k, r2.x, s.x);
      w.y *= born_ccf(k, r2.y, s.y);
    }
    bool ia = still_in<FULL>(v, k, r2.x, si, j0 + (j & 31));
    bool ib = still_in<FULL>(v, k, r2.y, si, j0 + ((j + 1) & 31));
    if (MASKED) {
      ia = ia && !((ex >> kk) & 1u);
      ib = ib && !((ex >> kk) & 2u);
    }
    if (MASKED || !FULL) {
      w.x = ia ? w.x : 0.f;
      w.y = ib ? w.y : 0.f;
    }
    GA = __ffma2_rn(w, make_float2(Q.z, Q.w), GA);
    GR = __ffma2_rn(w, VA, GR);
    ROT2(GR);
  }
  const float gr = GR.x + __shfl_sync(0xffffffffu, GR.y, (lane + 31) & 31), ga = GA.x + GA.y;
  fix_range(v.status, fabsf(ga) + fabsf(gr));
  atomic_add_ll(&gpol[si], fx32(ga));
  atomic_add_ll(&gpol[j0 + lane], fx32(gr));
}

// FAR: no pair of the item in close contact
template <bool FAR>
__device__ __forceinline__ void born_loop2(const DevView& v, const GBConst& k, int lane, int r0, const BornRows& rs,
                                           const float4& xa, const float4& xb, const float4& pa, const float4& pb,
                                           float c2, float2& GA, float2& GB, float2& GR) {
  const float2 AX = f2(-xa.x), AY = f2(-xa.y), AZ = f2(-xa.z), BX = f2(-xb.x), BY = f2(-xb.y), BZ = f2(-xb.z);
  const float2 VA = f2(k.born2 * pa.w), VB = f2(k.born2 * pb.w);
  const float4 *xy = rs.xy + lane, *zv = rs.zv + lane;
#pragma unroll 4
  for (int kk = 0; kk < 32; kk += 2) {
    const float4 P = xy[kk], Q = zv[kk];
    const float2 X = make_float2(P.x, P.y), Y = make_float2(P.z, P.w), Z = make_float2(Q.x, Q.y);
    const float2 VR = make_float2(Q.z, Q.w);
    const float2 ax = __fadd2_rn(X, AX), ay = __fadd2_rn(Y, AY), az = __fadd2_rn(Z, AZ);
    const float2 bx = __fadd2_rn(X, BX), by = __fadd2_rn(Y, BY), bz = __fadd2_rn(Z, BZ);
    const float2 ra = __ffma2_rn(az, az, __ffma2_rn(ay, ay, __fmul2_rn(ax, ax)));
    const float2 rb = __ffma2_rn(bz, bz, __ffma2_rn(by, by, __fmul2_rn(bx, bx)));
    const float2 ia = make_float2(rcp_ftz(ra.x), rcp_ftz(ra.y));
    const float2 ib = make_float2(rcp_ftz(rb.x), rcp_ftz(rb.y));
    float2 wa = __fmul2_rn(ia, ia), wb = __fmul2_rn(ib, ib);
    if (!FAR) {
      if (__any_sync(0xffffffffu, fminf(fminf(ra.x, ra.y), fminf(rb.x, rb.y)) <= c2)) {
        // rare: the rotating atoms' radii are read here, not staged
        const float R0 = v.par[r0 + ((lane + kk) & 31)].z, R1 = v.par[r0 + ((lane + kk + 1) & 31)].z;
        wa.x *= born_ccf(k, ra.x, pa.z + R0);
        wa.y *= born_ccf(k, ra.y, pa.z + R1);
        wb.x *= born_ccf(k, rb.x, pb.z + R0);
        wb.y *= born_ccf(k, rb.y, pb.z + R1);
      }
    }
    GA = __ffma2_rn(wa, VR, GA);
    GB = __ffma2_rn(wb, VR, GB);
    GR = __ffma2_rn(wa, VA, GR);
    GR = __ffma2_rn(wb, VB, GR);
    ROT2(GR);
  }
}

__device__ __forceinline__ void born_full2(const DevView& v, const GBConst& k, const Tile& A, const Tile& B, int lane,
                                           long long* gpol, BornRows& rs) {
  const int sa = A.bj * 32 + lane, sb = B.bj * 32 + lane, r0 = A.bi * 32;
  const int l1 = (lane + 1) & 31;
  const float4 xa = j_in_i_frame(v, A, lane), xb = j_in_i_frame(v, B, lane);
  const float4 pa = v.par[sa], pb = v.par[sb];
  const float4 x0 = v.xq[r0 + lane], x1 = v.xq[r0 + l1];
  const float4 p0 = v.par[r0 + lane], p1 = v.par[r0 + l1];
  __syncwarp();
  rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x1.x, x0.y, x1.y);
  rs.zv[lane] = rs.zv[lane + 32] = make_float4(x0.z, x1.z, k.born2 * p0.w, k.born2 * p1.w);
  __syncwarp();
  const float c2 = pair_contact2(k, make_float2(pa.z, pb.z), p0.z);
  float2 GA = f2(0.f), GB = f2(0.f), GR = f2(0.f);
  if (item_far(xa, xb, x0, c2, c2)) born_loop2<true>(v, k, lane, r0, rs, xa, xb, pa, pb, c2, GA, GB, GR);
  else born_loop2<false>(v, k, lane, r0, rs, xa, xb, pa, pb, c2, GA, GB, GR);
  // GR.x holds the sum of the rotating atom of this lane, GR.y that of lane + 1
  const float gr = GR.x + __shfl_sync(0xffffffffu, GR.y, (lane + 31) & 31);
  const float ga = GA.x + GA.y, gb = GB.x + GB.y;
  fix_range(v.status, fabsf(ga) + fabsf(gb) + fabsf(gr));
  atomic_add_ll(&gpol[sa], fx32(ga));
  atomic_add_ll(&gpol[sb], fx32(gb));
  atomic_add_ll(&gpol[r0 + lane], fx32(gr));
}

// ---------------------------------------------------------------------------
// pass 2: GB cross term fused with vacuum LJ + Coulomb, i > j pairs within Cutoff
// (forces, dE/da and, with ENERGY, the pair energies).
// ---------------------------------------------------------------------------
struct PairAcc {
  float fx, fy, fz, da;
};

// per-tile FP32 sums enter 64-bit fixed point before they are combined, so a
// slot's total does not depend on how its tiles were grouped into work items
__device__ __forceinline__ void flush_pair(const DevView& v, long long* deda, int s, const PairAcc& a) {
  fix_range(v.status, fabsf(a.fx) + fabsf(a.fy) + fabsf(a.fz) + fabsf(a.da));
  atomic_add_ll(&v.facc[force_at(s, 0)], fx32(a.fx));
  atomic_add_ll(&v.facc[force_at(s, 1)], fx32(a.fy));
  atomic_add_ll(&v.facc[force_at(s, 2)], fx32(a.fz));
  if (deda) atomic_add_ll(&deda[s], fx32(a.da));
}

// Born sums and the base law of an all-inside tile pair in one pass (the dynamics
// step's body): LJ and Coulomb at eps_out, which hold for every pair but those above the
// exp threshold (k_gb_pair adds what these differ by, once the radii are known).  Two
// passes used to walk every pair and form its distance; now the second walks a tenth of
// the items.  Each lane holds one atom of either j block (.x, .y), the i block's atoms
// come from the warp's rows.  Bound by the FMA pipe (56 of its cycles a step of two
// pairs a lane).  64 peptides (523 M pairs): Born 271 + pair 663 us -> 638 + 215 (half
// of it single tiles); one of 4,224 atoms 14.3 + 23.4 -> 20.7 + 18.0.  FAR: no pair of
// the item in close contact.
template <bool FAR>
__device__ __forceinline__ void born_base_loop2(const DevView& v, const GBConst& k, int lane, int r0, const BornRows& rs,
                                                const float4& xa, const float4& xb, const float4& pa, const float4& pb,
                                                float c2, float2& G, float2& FX, float2& FY, float2& FZ, float& gr,
                                                float3& R) {
  const float2 nx = make_float2(-xa.x, -xb.x), ny = make_float2(-xa.y, -xb.y), nz = make_float2(-xa.z, -xb.z);
  const float2 QN = make_float2(k.neg_sq_eout * xa.w, k.neg_sq_eout * xb.w), S = make_float2(pa.x, pb.x);
  const float2 EN = make_float2(-k.sqrt12 * pa.y, -k.sqrt12 * pb.y), V = make_float2(k.born2 * pa.w, k.born2 * pb.w);
  const float4 *x2 = rs.xy + lane, *p2 = rs.zv + lane;
#pragma unroll 2
  for (int kk = 0; kk < 32; kk++) {
    const float4 xr = x2[kk], pr = p2[kk];
    const float2 dx = __fadd2_rn(f2(xr.x), nx), dy = __fadd2_rn(f2(xr.y), ny), dz = __fadd2_rn(f2(xr.z), nz);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    const float2 QQ = __fmul2_rn(QN, f2(xr.w)), SS = __fadd2_rn(S, f2(pr.x)), EE = __fmul2_rn(EN, f2(pr.y));
    const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y)), i2 = make_float2(rcp_ftz(r2.x), rcp_ftz(r2.y));
    const float2 ir2 = __fmul2_rn(ir, ir);
    float2 w = __fmul2_rn(i2, i2);
    if (!FAR) {
      if (__any_sync(0xffffffffu, fminf(r2.x, r2.y) <= c2)) {
        const float R0 = v.par[r0 + ((lane + kk) & 31)].z;   // (rare: the radii are read here, not staged)
        w.x *= born_ccf(k, r2.x, pa.z + R0);
        w.y *= born_ccf(k, r2.y, pb.z + R0);
      }
    }
    G = __ffma2_rn(w, f2(pr.z), G);
    gr = fmaf(w.x, V.x, gr);
    gr = fmaf(w.y, V.y, gr);
    const float2 t2 = __fmul2_rn(__fmul2_rn(SS, SS), ir2);
    const float2 b6 = __fmul2_rn(__fmul2_rn(t2, t2), t2);
    const float2 amb = __fmul2_rn(b6, __fadd2_rn(b6, f2(-1.f)));
    const float2 g = __fmul2_rn(__ffma2_rn(EE, amb, __fmul2_rn(QQ, ir)), ir2);
    FX = __ffma2_rn(g, dx, FX);
    FY = __ffma2_rn(g, dy, FY);
    FZ = __ffma2_rn(g, dz, FZ);
    R.x = fmaf(g.x, dx.x, R.x); R.x = fmaf(g.y, dx.y, R.x);
    R.y = fmaf(g.x, dy.x, R.y); R.y = fmaf(g.y, dy.y, R.y);
    R.z = fmaf(g.x, dz.x, R.z); R.z = fmaf(g.y, dz.y, R.z);
    ROT(gr); ROT(R.x); ROT(R.y); ROT(R.z);
  }
}

__device__ __forceinline__ void born_base_full2(const DevView& v, const GBConst& k, const Tile& A, const Tile& B, int lane,
                                                long long* gpol, BornRows& rs) {
  const int sa = A.bj * 32 + lane, sb = B.bj * 32 + lane, r0 = A.bi * 32;
  const float4 xa = j_in_i_frame(v, A, lane), xb = j_in_i_frame(v, B, lane);
  const float4 pa = v.par[sa], pb = v.par[sb], x0 = v.xq[r0 + lane], p0 = v.par[r0 + lane];
  __syncwarp();
  rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x0.y, x0.z, k.sq_eout * x0.w);
  rs.zv[lane] = rs.zv[lane + 32] = make_float4(p0.x, k.sqrt12 * p0.y, k.born2 * p0.w, 0.f);
  __syncwarp();
  const float c2 = pair_contact2(k, make_float2(pa.z, pb.z), p0.z);
  float2 G = f2(0.f), FX = f2(0.f), FY = f2(0.f), FZ = f2(0.f);
  float gr = 0.f;
  float3 R = make_float3(0.f, 0.f, 0.f);   // minus the rotating atom's force
  if (item_far(xa, xb, x0, c2, c2)) born_base_loop2<true>(v, k, lane, r0, rs, xa, xb, pa, pb, c2, G, FX, FY, FZ, gr, R);
  else born_base_loop2<false>(v, k, lane, r0, rs, xa, xb, pa, pb, c2, G, FX, FY, FZ, gr, R);
  fix_range(v.status, fabsf(G.x) + fabsf(G.y) + fabsf(gr));
  atomic_add_ll(&gpol[sa], fx32(G.x));
  atomic_add_ll(&gpol[sb], fx32(G.y));
  atomic_add_ll(&gpol[r0 + lane], fx32(gr));
  flush_pair(v, nullptr, sa, PairAcc{FX.x, FY.x, FZ.x, 0.f});
  flush_pair(v, nullptr, sb, PairAcc{FX.y, FY.y, FZ.y, 0.f});
  flush_pair(v, nullptr, r0 + lane, PairAcc{-R.x, -R.y, -R.z, 0.f});
}

// whether both tiles of a work item are all inside, by their flags or (gradient
// calls, whose lists carry none) at run time
__device__ __forceinline__ bool pair_full_now(const DevView& v, const GBConst& k, const Tile& T, const Tile& U,
                                              int lane) {
  if (tile_full(T) && tile_full(U)) return true;
  if (k.far_inner <= 0.f) return false;
  const float4 x = v.xq[T.bi * 32 + lane];
  return tile_full_now(k, T, x, j_in_i_frame(v, T, lane)) && tile_full_now(k, U, x, j_in_i_frame(v, U, lane));
}

__device__ __forceinline__ void born_single(const DevView& v, const GBConst& k, const Tile& T, int lane,
                                            long long* gpol, BornRows& rs) {
  const bool full = tile_full_now(k, T, v.xq[T.bi * 32 + lane], j_in_i_frame(v, T, lane));
  if (tile_masked(T)) {
    unsigned ex, m14;
    tile_masks(v, T, lane, ex, m14);
    if (T.flags & 2) ex |= diag_exclusion(lane);
    if (full) born_tile<true, true>(v, k, T, lane, ex, gpol, rs);
    else born_tile<true, false>(v, k, T, lane, ex, gpol, rs);
  } else if (full) {
    born_tile<false, true>(v, k, T, lane, 0u, gpol, rs);
  } else {
    born_tile<false, false>(v, k, T, lane, 0u, gpol, rs);
  }
}

// BASE: with the base law's forces of all-inside tile pairs (force-only FastMode passes);
// six CTAs of 128 threads an SM (five: 657 us on the 64 peptides)
constexpr int kBaseThreads = 128;
template <bool BASE>
__global__ void __launch_bounds__(BASE ? kBaseThreads : kBornThreads, BASE ? 6 : 5)
    k_gb_born(const __grid_constant__ DevView v, const __grid_constant__ GBConst k, long long* gpol) {
  pdl_sync();
  __shared__ BornRows rows[(BASE ? kBaseThreads : kBornThreads) / 32];
  BornRows& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int ni = *v.nitems;
  for (int it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < ni; it += nwarps) {
    const int2 t = v.items[it];
    const Tile T = v.tiles[t.x];
    if (t.y >= 0) {
      const Tile U = v.tiles[t.y];
      if (BASE && tile_full(T) && tile_full(U)) {
        born_base_full2(v, k, T, U, lane, gpol, rs);
        continue;
      }
      if (pair_full_now(v, k, T, U, lane)) {
        born_full2(v, k, T, U, lane, gpol, rs);
        continue;
      }
      born_single(v, k, U, lane, gpol, rs);
    }
    born_single(v, k, T, lane, gpol, rs);
  }
}

// Born radii a = -halfeconv / (terms123 + sum) + BornRadiusOffset  (FP64)
__global__ void k_gb_radii(DevView v, const double* terms123, const long long* gpol, double gscale, double halfeconv,
                           double offset, float* born_f, double* born_d, float* bborn) {
  pdl_sync();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= v.nslots) return;   // (whole warps)
  int a = v.sorted_atom[s];
  float f = 1.f;
  if (a >= 0) {
    double G = terms123[a] + (double)gpol[s] * gscale;
    double r = -halfeconv / G + offset;
    f = (float)r;
    born_d[a] = r;
  }
  born_f[s] = f;
  f = fabsf(f);   // (a non-finite radius leaves no bound: every item is looked at)
  if (!(f < 3.0e38f)) f = 3.0e38f;
  f = warp_max(f);
  if ((s & 31) == 0) bborn[s >> 5] = f;
}

// Two pairs of the fused law on packed FP32x2 arithmetic.  In: r^2, the products
// QQ = -econv_out q q (ENERGY: -q q), EE = -12 eps, AA = K a a, (ENERGY) aa = a a, and
// the LJ radius sums SS.  Common pair: vacuum LJ + Coulomb at eps_out, dE/dr / r = -(12 eps (A - B)
// + E_out) / r^2, whose bracket is one FFMA.  A pair with r^2 <= AA may lie
// above the exp threshold; when any lane of the warp has one (a vote), the GB
// term (gbff.cpp:1592-1678) is formed for both halves, with Coulomb at eps_in in
// place of eps_out, and zeroed where the exact decision (FP64 within rounding of
// the threshold) says no.
//   MASKED: pa, pb: the pair counts at all (diagonal); xa, xb: bond order <= 2
//     (GB term only); s14: 1-4 (vdw14 / elec14 scaling)
//   FULL: inside every cutoff and switch radius
//   FAST: the vacuum terms are part of the law (FastMode); else the GB term
//     alone, premul q q / r below the threshold (calcBornForces, :1308-1325)
struct Mask2 {
  bool pa, pb, xa, xb, ma, mb;
};
// out: g = dE/dr / r (force on the held atom along d), W = dE/da per unit of the
// partner's radius (zero unless `any`), and with ENERGY the pairs' energies: vdW,
// Coulomb per econv_out, GB cross term per 2 premul (a constant in FP32, or products
// with it, would shift all of them alike: it meets their sums in double-float)
struct Pair2 {
  float2 g, W, ev, ee, ep;
  bool any;
};

template <bool MASKED, bool FULL, bool FAST, bool ENERGY>
__device__ __forceinline__ Pair2 gb_pair2(const DevView& v, const GBConst& k, float2 r2, float2 QQ, float2 SS,
                                          float2 EE, float2 AA, float2 aa, const Mask2& m, int ha, int hb, int ra,
                                          int rb) {
  Pair2 o;
  const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 ir2 = __fmul2_rn(ir, ir);
  const bool ina = (FULL || r2.x <= k.cut2) && (!MASKED || m.pa);
  const bool inb = (FULL || r2.y <= k.cut2) && (!MASKED || m.pb);
  float2 e1 = __fmul2_rn(QQ, ir);   // -E_out (ENERGY: per econv_out)
  // switching without a branch: below the inner cutoff w = 0 gives S = 1 and dS = 0 exactly
  float2 S = f2(1.f), dS = f2(0.f), r = f2(0.f);
  if (!FULL) {
    r = __fmul2_rn(r2, ir);
    const float2 w = make_float2(fmaxf(r.x - k.inner, 0.f), fmaxf(r.y - k.inner, 0.f));
    const float2 wi = __fmul2_rn(w, f2(-k.invw2));
    const float2 sw = __ffma2_rn(w, wi, f2(1.f));
    dS = __fmul2_rn(__fmul2_rn(wi, sw), f2(4.f));
    S = __fmul2_rn(sw, sw);
  }
  float2 vb = f2(0.f), ev = f2(0.f);   // -12 eps (A - B), eps (A - 2B)
  if (FAST) {
    if (MASKED) {
      EE = __fmul2_rn(EE, make_float2(m.ma ? k.vdw14 : 1.f, m.mb ? k.vdw14 : 1.f));
      e1 = __fmul2_rn(e1, make_float2(m.ma ? k.elec14 : 1.f, m.mb ? k.elec14 : 1.f));
    }
    const float2 t2 = __fmul2_rn(__fmul2_rn(SS, SS), ir2);
    const float2 b6 = __fmul2_rn(__fmul2_rn(t2, t2), t2);
    const float2 amb = __ffma2_rn(b6, b6, __fmul2_rn(b6, f2(-1.f)));
    vb = __fmul2_rn(EE, amb);
    if (ENERGY || !FULL) ev = __fmul2_rn(__ffma2_rn(EE, __fmul2_rn(b6, f2(-1.f)), vb), f2(-1.f / 12.f));
    if (MASKED) {
      vb = make_float2(m.xa ? 0.f : vb.x, m.xb ? 0.f : vb.y);
      e1 = make_float2(m.xa ? 0.f : e1.x, m.xb ? 0.f : e1.y);
      if (ENERGY || !FULL) ev = make_float2(m.xa ? 0.f : ev.x, m.xb ? 0.f : ev.y);
    }
  }
  o.W = f2(0.f);
  if (ENERGY) o.ep = f2(0.f);
  float2 gg = f2(0.f);
  const bool na = ina && r2.x <= AA.x, nb = inb && r2.y <= AA.y;
  o.any = __any_sync(0xffffffffu, na || nb);
  bool ona = false, onb = false;
  if (o.any) {
    if (!ENERGY) aa = __fmul2_rn(AA, f2(k.invK));
    const float2 rc = ENERGY ? make_float2(rcp_ftz(aa.x), rcp_ftz(aa.y)) : make_float2(rcp_ftz(AA.x), rcp_ftz(AA.y));
    const float2 u = __fmul2_rn(__fmul2_rn(r2, rc), f2(ENERGY ? -0.25f : k.kU));
    const float tie = 2e-6f * fabsf(k.thresh);
    ona = na && u.x > k.thresh;
    onb = nb && u.y > k.thresh;
    if (na && fabsf(u.x - k.thresh) <= tie) ona = gb_on_fp64(v, ha, ra, k.thresh_d);
    if (nb && fabsf(u.y - k.thresh) <= tie) onb = gb_on_fp64(v, hb, rb, k.thresh_d);
    const float2 tg = make_float2(__expf(u.x), __expf(u.y));
    const float2 D = __ffma2_rn(tg, aa, r2);
    const float2 fgb = make_float2(rsqrtf(D.x), rsqrtf(D.y));
    float2 ep = ENERGY ? __fmul2_rn(QQ, fgb) : __fmul2_rn(__fmul2_rn(QQ, f2(k.gb_ep)), fgb);
    ep = make_float2(ona ? ep.x : 0.f, onb ? ep.y : 0.f);
    if (ENERGY) {
      o.ep = __fmul2_rn(__fmul2_rn(ep, S), f2(-1.f));
      ep = __fmul2_rn(ep, f2(-k.premul));
    }
    float2 w = __fmul2_rn(ep, __fmul2_rn(fgb, fgb));
    if (!FULL) w = __fmul2_rn(w, S);
    gg = __fmul2_rn(w, __ffma2_rn(tg, f2(0.5f), f2(-2.f)));                   // 2 dE/dr / r
    if (!FULL) gg = __ffma2_rn(__fmul2_rn(__fmul2_rn(ep, dS), f2(2.f)), ir, gg);
    o.W = __fmul2_rn(__fmul2_rn(w, tg), __fadd2_rn(u, f2(-1.f)));             // -ep tg (1 - u) l
    if (FAST) e1 = make_float2(ona ? e1.x * k.in_over_out : e1.x, onb ? e1.y * k.in_over_out : e1.y);
  }
  if (!FAST) {
    float2 ep = ENERGY ? __fmul2_rn(QQ, ir) : __fmul2_rn(__fmul2_rn(QQ, f2(k.gb_ep)), ir);
    ep = make_float2(ona || !ina ? 0.f : ep.x, onb || !inb ? 0.f : ep.y);
    if (ENERGY) {
      o.ep = __ffma2_rn(__fmul2_rn(ep, f2(-1.f)), S, o.ep);
      ep = __fmul2_rn(ep, f2(-k.premul));
    }
    gg = __ffma2_rn(__fmul2_rn(__fmul2_rn(ep, S), f2(-2.f)), ir2, gg);
    gg = __ffma2_rn(__fmul2_rn(__fmul2_rn(ep, dS), f2(2.f)), ir, gg);
    o.g = gg;
    if (MASKED || !FULL) o.g = make_float2(ina ? o.g.x : 0.f, inb ? o.g.y : 0.f);
    return o;
  }
  if (ENERGY) {
    o.ee = __fmul2_rn(e1, f2(-1.f));
    e1 = __fmul2_rn(e1, f2(k.eout));
  }
  if (FULL) {
    o.g = __ffma2_rn(__fadd2_rn(vb, e1), ir2, gg);
    if (ENERGY) o.ev = ev;
  } else {
    const float2 w = make_float2(fmaxf(r.x - k.vdwinner, 0.f), fmaxf(r.y - k.vdwinner, 0.f));
    const float2 wi = __fmul2_rn(w, f2(-k.vdwinvw2));
    const float2 sw = __ffma2_rn(w, wi, f2(1.f));
    const bool va = r.x < k.vdwcut, vb_ = r.y < k.vdwcut;
    float2 Sv = __fmul2_rn(sw, sw), dSv = __fmul2_rn(__fmul2_rn(wi, sw), f2(4.f));
    Sv = make_float2(va ? Sv.x : 0.f, vb_ ? Sv.y : 0.f);
    dSv = make_float2(va ? dSv.x : 0.f, vb_ ? dSv.y : 0.f);
    const float2 b = __ffma2_rn(Sv, vb, __fmul2_rn(S, e1));
    const float2 d = __ffma2_rn(ev, dSv, __fmul2_rn(__fmul2_rn(e1, f2(-1.f)), dS));
    o.g = __ffma2_rn(b, ir2, __ffma2_rn(d, ir, gg));
    if (ENERGY) {
      o.ev = __fmul2_rn(ev, Sv);
      o.ee = __fmul2_rn(o.ee, S);
    }
  }
  if (MASKED || !FULL) {   // (a select, not a product: the diagonal's own pair has r = 0)
    o.g = make_float2(ina ? o.g.x : 0.f, inb ? o.g.y : 0.f);
    if (ENERGY) {
      o.ev = make_float2(ina ? o.ev.x : 0.f, inb ? o.ev.y : 0.f);
      o.ee = make_float2(ina ? o.ee.x : 0.f, inb ? o.ee.y : 0.f);
    }
  }
  return o;
}

// ---------------------------------------------------------------------------
// Pair energies (ENERGY passes).  The vdW total is a small difference of large
// repulsive and attractive sums: FP32 positions (rounded relative to their block
// centres) on the close contacts, or FP32 sums, leave ~1e-6 of it.  So pairs
// closer than sqrt(GBConst::eclose2) (4.5 A: the close contacts that carry the
// large repulsive terms) are left out of the FP32 sums and listed, and their
// energies formed in double-float from double-float positions and parameters,
// the list dealt over the lanes; the other pairs' energies are the FP32 terms,
// summed over 8 rotation steps and then in double-float.  A tile's sums meet over
// the warp in double-float and enter fixed point once.  The displacements of these
// passes are differences of double-float positions rounded once to FP32, so their
// forces carry no rounding of the block frames (6e-7 of them, 1.2e-6 without), and the
// close pairs' r^2 are rounded once (close_r2).
// ---------------------------------------------------------------------------
// the rotating block in the warp's shared memory: single tiles as step pairs
// (x, x', y, y'), (z, z', q, q'), (LJ radius, ', sqrt(eps), ') and (Born radius, x
// sqrtK in the force-only passes, '); tile pairs as (x, y, z, q sqrt(econv_out)) and
// Born radii x sqrtK, twice over, so that a lane's row at step kk lies at a fixed offset
struct PairRows {
  union {
    struct {
      float4 xy[32], zq[32], se[32];
      float2 ak[32];
    };
    struct {
      float4 x2[64], p2[64];
    };
  };
};
struct PairRowsE : PairRows {
  float4 lxy[32];                  // what FP32 rounding takes off (x, x', y, y')
  float2 lz[32];                   // and (z, z')
  unsigned short pair[1024];       // i lane | j row << 5 | bond order <= 2 << 10 | 1-4 << 11
};

// (ENERGY) energies of one listed close pair into the sums
struct GBESum {
  DF v, e, p;
};
template <bool FAST>
__device__ __forceinline__ void gb_close_energy(const DevView& v, const GBConst& k, const Tile& T, const DF O[3],
                                                unsigned code, const float* born, GBESum& sum) {
  const int si = T.bi * 32 + (code & 31), sj = T.bj * 32 + ((code >> 5) & 31);
  const bool excl = code & 1024u, is14 = code & 2048u;
  const float4 xh = v.xq[si], xl = v.rlo[si], yh = v.xq[sj], yl = v.rlo[sj], pi = v.par[si], pj = v.par[sj];
  const float2 pil = v.plo[si], pjl = v.plo[sj];
  const DF dx = df_sub(df_add(DF{yh.x, yl.x}, O[0]), DF{xh.x, xl.x});
  const DF dy = df_sub(df_add(DF{yh.y, yl.y}, O[1]), DF{xh.y, xl.y});
  const DF dz = df_sub(df_add(DF{yh.z, yl.z}, O[2]), DF{xh.z, xl.z});
  const DF r2 = df_norm2(dx, dy, dz);
  const DF ir = df_rsqrt(r2);
  const float r = r2.h * ir.h;
  const float ai = born[si], aj = born[sj];
  const float u = -0.25f * __fdividef(r2.h, ai * aj);
  bool on = u > k.thresh;
  if (fabsf(u - k.thresh) <= 2e-6f * fabsf(k.thresh)) on = gb_on_fp64(v, si, sj, k.thresh_d);
  const float w = fmaxf(r - k.inner, 0.f), sw = 1.f - w * w * k.invw2, S = sw * sw;
  const DF qq = df_norm(df_mul(DF{xh.w, xl.w}, DF{yh.w, yl.w}));
  const DF c = df_norm(df_mul(qq, ir));
  if (on) {
    const float fgb = rsqrtf(fmaf(__expf(u), ai * aj, r2.h));
    df_acc(sum.p, df_norm(df_scale(df_mul(k.premul2_f, qq), fgb * S)));
  } else if (!FAST) {
    df_acc(sum.p, df_norm(df_scale(df_mul(k.premul2_f, c), S)));
  }
  if (FAST && !excl) {
    DF E = df_norm(df_mul(on ? k.econv_in_f : k.econv_out_f, c));
    if (is14) E = df_norm(df_mul(E, k.elec14_f));
    df_acc(sum.e, df_norm(df_scale(E, S)));
    const DF R = df_norm(df_add(DF{pi.x, pil.x}, DF{pj.x, pjl.x}));
    const DF t = df_norm(df_mul(R, ir)), t2 = df_norm(df_mul(t, t));
    const DF B = df_norm(df_mul(df_mul(t2, t2), t2));
    DF eps = df_norm(df_mul(DF{pi.y, pil.y}, DF{pj.y, pjl.y}));
    if (is14) eps = df_norm(df_mul(eps, k.vdw14_f));
    const float wv = fmaxf(r - k.vdwinner, 0.f), sv = 1.f - wv * wv * k.vdwinvw2;
    const float Sv = r < k.vdwcut ? sv * sv : 0.f;
    df_acc(sum.v, df_norm(df_scale(df_mul(eps, df_norm(df_sub(df_mul(B, B), df_scale2(B, 2.f)))), Sv)));
  }
}

// (ENERGY) r^2 of two steps' pairs rounded once, from the displacements' exact high parts
// p + x and low parts l; the displacements rounded once into d.  The repulsion of a close
// pair goes with r^-14: the two or three roundings of a plain sum of squares were most of
// its force's error.
__device__ __forceinline__ float2 close_r2(float2 px, float2 x, float2 lx, float2 py, float2 y, float2 ly, float2 pz,
                                           float2 z, float2 lz, float2& dx, float2& dy, float2& dz) {
  auto exact = [](float2 p, float2 x, float2 l, float2& d) {
    DF2 s = df_two_sum(p, x);
    s = df_fast_two_sum(s.h, __fadd2_rn(s.l, l));
    d = s.h;
    return s;
  };
  const DF2 a = exact(px, x, lx, dx), b = exact(py, y, ly, dy), c = exact(pz, z, lz, dz);
  return df_norm2(a, b, c).h;
}

// Pair pass of a single tile, step-packed: lane l holds i atom l (its values in
// both halves), the j block's atoms l + kk and l + kk + 1 come from the warp's
// rows; the rotating atoms' sums move two lanes per step.
template <bool MASKED, bool FULL, bool FAST, bool ENERGY>
__device__ __forceinline__ void gb_pair_tile(const DevView& v, const GBConst& k, const Tile& T, int lane,
                                             const float* born, long long* deda, PairRows& rs, PairRowsE* re) {
  const int si = T.bi * 32 + lane, j0 = T.bj * 32, l1 = (lane + 1) & 31;
  const float4 xi = v.xq[si], pi = v.par[si];
  DF O[3];                 // (ENERGY) centre of bj seen from bi
  float O0[3];             // (open space: nothing left)
  float2 XL, YL, ZL;       // remainders of the held atom, negated
  unsigned ex = 0u, m14 = 0u, dm = 0u;
  if (MASKED) {
    tile_masks(v, T, lane, ex, m14);
    dm = (T.flags & 2) ? diag_exclusion(lane) : 0u;
  }
  {
    float4 x0 = j_in_i_frame(v, T, lane);
    const float4 p0 = v.par[j0 + lane];
    if (ENERGY) {
      const float o[3] = {T.ox, T.oy, T.oz};
      df_offset(v, v.sys[v.slot_sys[T.bi]], T.bi, T.bj, o, O, O0);
      const float4 h = v.xq[j0 + lane], l = v.rlo[j0 + lane], li = v.rlo[si];
      const DF jx = df_norm(df_add(DF{h.x, l.x}, O[0])), jy = df_norm(df_add(DF{h.y, l.y}, O[1]));
      const DF jz = df_norm(df_add(DF{h.z, l.z}, O[2]));
      x0.x = jx.h;
      x0.y = jy.h;
      x0.z = jz.h;
      const float x1 = __shfl_sync(0xffffffffu, jx.l, l1), y1 = __shfl_sync(0xffffffffu, jy.l, l1);
      const float z1 = __shfl_sync(0xffffffffu, jz.l, l1);
      __syncwarp();
      re->lxy[lane] = make_float4(jx.l, x1, jy.l, y1);
      re->lz[lane] = make_float2(jz.l, z1);
      XL = f2(-li.x);
      YL = f2(-li.y);
      ZL = f2(-li.z);
    }
    const float q0 = x0.w, e0 = p0.y, a0 = (ENERGY ? 1.f : k.sqrtK) * born[j0 + lane];
    const float x1 = __shfl_sync(0xffffffffu, x0.x, l1), y1 = __shfl_sync(0xffffffffu, x0.y, l1);
    const float z1 = __shfl_sync(0xffffffffu, x0.z, l1), q1 = __shfl_sync(0xffffffffu, q0, l1);
    const float s1 = __shfl_sync(0xffffffffu, p0.x, l1), e1 = __shfl_sync(0xffffffffu, e0, l1);
    const float a1 = __shfl_sync(0xffffffffu, a0, l1);
    __syncwarp();
    rs.xy[lane] = make_float4(x0.x, x1, x0.y, y1);
    rs.zq[lane] = make_float4(x0.z, z1, q0, q1);
    rs.se[lane] = make_float4(p0.x, s1, e0, e1);
    rs.ak[lane] = make_float2(a0, a1);
    __syncwarp();
  }
  const float2 X = f2(-xi.x), Y = f2(-xi.y), Z = f2(-xi.z), Q = f2(ENERGY ? -xi.w : -k.eout * xi.w), R = f2(pi.x);
  const float2 E = f2(-12.f * pi.y), AK = f2((ENERGY ? 1.f : k.sqrtK) * born[si]);
  float2 FX = f2(0.f), FY = f2(0.f), FZ = f2(0.f), DA = f2(0.f);
  float2 RX = f2(0.f), RY = f2(0.f), RZ = f2(0.f), RA = f2(0.f);   // minus the rotating atoms' forces; their dE/da
  float2 cv = f2(0.f), ce = f2(0.f), cp = f2(0.f);                 // (ENERGY) FP32 sums of 8 steps
  GBESum sum = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  int np = 0;
#pragma unroll 1
  for (int kk = 0; kk < 32; kk += 2) {
    const int j = (lane + kk) & 31;
    const float4 P = rs.xy[j], ZQ = rs.zq[j], SE = rs.se[j];
    const float2 ak = rs.ak[j];
    float2 dx = __fadd2_rn(make_float2(P.x, P.y), X), dy = __fadd2_rn(make_float2(P.z, P.w), Y);
    float2 dz = __fadd2_rn(make_float2(ZQ.x, ZQ.y), Z);
    float2 lx, ly, lz;
    if (ENERGY) {
      const float4 L = re->lxy[j];
      lx = __fadd2_rn(make_float2(L.x, L.y), XL);
      ly = __fadd2_rn(make_float2(L.z, L.w), YL);
      lz = __fadd2_rn(re->lz[j], ZL);
      dx = __fadd2_rn(dx, lx);
      dy = __fadd2_rn(dy, ly);
      dz = __fadd2_rn(dz, lz);
    }
    float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    Mask2 m = {true, true, false, false, false, false};
    if (MASKED) {
      m.pa = !((dm >> kk) & 1u);
      m.pb = !((dm >> kk) & 2u);
      m.xa = (ex >> kk) & 1u;
      m.xb = (ex >> kk) & 2u;
      m.ma = (m14 >> kk) & 1u;
      m.mb = (m14 >> kk) & 2u;
    }
    bool ca = false, cb = false, close = false;
    if (ENERGY) {
      ca = r2.x < k.eclose2 && (FULL || r2.x <= k.cut2) && m.pa;
      cb = r2.y < k.eclose2 && (FULL || r2.y <= k.cut2) && m.pb;
      close = __any_sync(0xffffffffu, ca || cb);
      if (close)
        r2 = close_r2(make_float2(P.x, P.y), X, lx, make_float2(P.z, P.w), Y, ly, make_float2(ZQ.x, ZQ.y), Z, lz, dx, dy, dz);
    }
    const float2 AA = __fmul2_rn(AK, ak);
    const Pair2 o = gb_pair2<MASKED, FULL, FAST, ENERGY>(
        v, k, r2, __fmul2_rn(Q, make_float2(ZQ.z, ZQ.w)), __fadd2_rn(R, make_float2(SE.x, SE.y)),
        __fmul2_rn(E, make_float2(SE.z, SE.w)), ENERGY ? __fmul2_rn(AA, f2(k.K)) : AA, AA, m, si, si, j0 + j,
        j0 + ((j + 1) & 31));
    FX = __ffma2_rn(o.g, dx, FX); FY = __ffma2_rn(o.g, dy, FY); FZ = __ffma2_rn(o.g, dz, FZ);
    RX = __ffma2_rn(o.g, dx, RX); RY = __ffma2_rn(o.g, dy, RY); RZ = __ffma2_rn(o.g, dz, RZ);
    if (o.any) {
      DA = __ffma2_rn(o.W, ak, DA);
      RA = __ffma2_rn(o.W, AK, RA);
    }
    ROT2(RX); ROT2(RY); ROT2(RZ); ROT2(RA);
    if (ENERGY) {
      float2 f = f2(1.f);
      if (close) {
        const unsigned ma = __ballot_sync(0xffffffffu, ca), mb = __ballot_sync(0xffffffffu, cb);
        const unsigned lt = (1u << lane) - 1u;
        if (ca)
          re->pair[np + __popc(ma & lt)] = (unsigned short)(lane | (j << 5) | (m.xa ? 1024 : 0) | (m.ma ? 2048 : 0));
        np += __popc(ma);
        if (cb)
          re->pair[np + __popc(mb & lt)] =
              (unsigned short)(lane | (((j + 1) & 31) << 5) | (m.xb ? 1024 : 0) | (m.mb ? 2048 : 0));
        np += __popc(mb);
        f = make_float2(ca ? 0.f : 1.f, cb ? 0.f : 1.f);
      }
      if (FAST) {
        cv = __ffma2_rn(f, o.ev, cv);
        ce = __ffma2_rn(f, o.ee, ce);
      }
      cp = __ffma2_rn(f, o.ep, cp);
      if ((kk & 6) == 6) {
        if (FAST) {
          df_acc(sum.v, df_two_sum(cv.x, cv.y));
          df_acc(sum.e, df_two_sum(ce.x, ce.y));
        }
        df_acc(sum.p, df_two_sum(cp.x, cp.y));
        cv = ce = cp = f2(0.f);
      }
    }
  }
  const int lm = (lane + 31) & 31;
  const float rx = RX.x + __shfl_sync(0xffffffffu, RX.y, lm), ry = RY.x + __shfl_sync(0xffffffffu, RY.y, lm);
  const float rz = RZ.x + __shfl_sync(0xffffffffu, RZ.y, lm), ra = RA.x + __shfl_sync(0xffffffffu, RA.y, lm);
  const float ia = ENERGY ? 1.f : k.inv_sqrtK;
  flush_pair(v, deda, si, PairAcc{FX.x + FX.y, FY.x + FY.y, FZ.x + FZ.y, (DA.x + DA.y) * ia});
  flush_pair(v, deda, j0 + lane, PairAcc{-rx, -ry, -rz, ra * ia});
  if (ENERGY) {
    if (FAST) sum.e = df_norm(df_mul(sum.e, k.eout_f));
    sum.p = df_norm(df_mul(sum.p, k.premul2_f));
    __syncwarp();
    for (int p = lane; p < np; p += 32) gb_close_energy<FAST>(v, k, T, O, re->pair[p], born, sum);
    __syncwarp();
    const DF e0 = df_warp_sum(sum.v), e1 = df_warp_sum(sum.e), e2 = df_warp_sum(sum.p);
    const DF x = lane == 0 ? e0 : (lane == 1 ? e1 : e2);
    if (lane < 3) {
      long long* En = v.eacc + (size_t)v.slot_sys[T.bi] * E_NSLOTS;
      atomic_add_ll(&En[lane == 0 ? E_VDW : (lane == 1 ? E_ELEC : E_POL_CROSS)],
                    fix_energy_d((double)x.h + (double)x.l));
    }
  }
}

// What pairs above the exp threshold have beyond the base law (k_gb_born): Coulomb at
// eps_in for eps_out, the GB term and its dE/da (QQ, AA as gb_pair2).  Zero, and any
// false, where no lane has such a pair.
__device__ __forceinline__ float2 gb_near2(const DevView& v, const GBConst& k, float2 r2, float2 QQ, float2 AA, int ha,
                                           int hb, int r, float2& W, bool& any) {
  const bool na = r2.x <= AA.x, nb = r2.y <= AA.y;
  any = __any_sync(0xffffffffu, na || nb);
  if (!any) return f2(0.f);
  const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 rc = make_float2(rcp_ftz(AA.x), rcp_ftz(AA.y));
  const float2 u = __fmul2_rn(__fmul2_rn(r2, rc), f2(k.kU));
  const float tie = 2e-6f * fabsf(k.thresh);
  bool ona = na && u.x > k.thresh, onb = nb && u.y > k.thresh;
  if (na && fabsf(u.x - k.thresh) <= tie) ona = gb_on_fp64(v, ha, r, k.thresh_d);
  if (nb && fabsf(u.y - k.thresh) <= tie) onb = gb_on_fp64(v, hb, r, k.thresh_d);
  QQ = make_float2(ona ? QQ.x : 0.f, onb ? QQ.y : 0.f);
  const float2 tg = make_float2(__expf(u.x), __expf(u.y));
  const float2 D = __ffma2_rn(tg, __fmul2_rn(AA, f2(k.invK)), r2);
  const float2 fgb = make_float2(rsqrtf(D.x), rsqrtf(D.y));
  const float2 w = __fmul2_rn(__fmul2_rn(__fmul2_rn(QQ, f2(k.gb_ep)), fgb), __fmul2_rn(fgb, fgb));
  const float2 gg = __fmul2_rn(w, __ffma2_rn(tg, f2(0.5f), f2(-2.f)));
  W = __fmul2_rn(__fmul2_rn(w, tg), __fadd2_rn(u, f2(-1.f)));
  const float2 e1 = __fmul2_rn(__fmul2_rn(QQ, ir), f2(k.in_over_out - 1.f));
  return __ffma2_rn(e1, __fmul2_rn(ir, ir), gg);
}

// those of an all-inside tile pair: the shape of born_base_full2
__device__ __forceinline__ void gb_near_full2(const DevView& v, const GBConst& k, const Tile& A, const Tile& B, int lane,
                                              const float* born, long long* deda, PairRows& rs) {
  const int sa = A.bj * 32 + lane, sb = B.bj * 32 + lane, r0 = A.bi * 32;
  const float4 xa = j_in_i_frame(v, A, lane), xb = j_in_i_frame(v, B, lane), x0 = v.xq[r0 + lane];
  const float2 AK = make_float2(k.sqrtK * born[sa], k.sqrtK * born[sb]);
  const float a0 = k.sqrtK * born[r0 + lane], akm = warp_max(a0) * 1.00001f;
  if (item_far(xa, xb, x0, AK.x * akm, AK.y * akm)) return;
  float* ar = reinterpret_cast<float*>(rs.p2);
  __syncwarp();
  rs.x2[lane] = rs.x2[lane + 32] = make_float4(x0.x, x0.y, x0.z, k.sq_eout * x0.w);
  ar[lane] = ar[lane + 32] = a0;
  __syncwarp();
  const float2 nx = make_float2(-xa.x, -xb.x), ny = make_float2(-xa.y, -xb.y), nz = make_float2(-xa.z, -xb.z);
  const float2 QN = make_float2(k.neg_sq_eout * xa.w, k.neg_sq_eout * xb.w);
  float2 FX = f2(0.f), FY = f2(0.f), FZ = f2(0.f), DA = f2(0.f);
  PairAcc R = {0.f, 0.f, 0.f, 0.f};   // minus the rotating atom's force; its dE/da
#pragma unroll 2
  for (int kk = 0; kk < 32; kk++) {
    const float4 xr = rs.x2[lane + kk];
    const float ak = ar[lane + kk];
    const float2 dx = __fadd2_rn(f2(xr.x), nx), dy = __fadd2_rn(f2(xr.y), ny), dz = __fadd2_rn(f2(xr.z), nz);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    float2 W;
    bool any;
    const float2 g = gb_near2(v, k, r2, __fmul2_rn(QN, f2(xr.w)), __fmul2_rn(AK, f2(ak)), sa, sb,
                              r0 + ((lane + kk) & 31), W, any);
    if (any) {
      FX = __ffma2_rn(g, dx, FX);
      FY = __ffma2_rn(g, dy, FY);
      FZ = __ffma2_rn(g, dz, FZ);
      DA = __ffma2_rn(W, f2(ak), DA);
      R.fx = fmaf(g.x, dx.x, R.fx); R.fx = fmaf(g.y, dx.y, R.fx);
      R.fy = fmaf(g.x, dy.x, R.fy); R.fy = fmaf(g.y, dy.y, R.fy);
      R.fz = fmaf(g.x, dz.x, R.fz); R.fz = fmaf(g.y, dz.y, R.fz);
      R.da = fmaf(W.x, AK.x, R.da);
      R.da = fmaf(W.y, AK.y, R.da);
    }
    ROT(R.fx); ROT(R.fy); ROT(R.fz); ROT(R.da);
  }
  flush_pair(v, deda, sa, PairAcc{FX.x, FY.x, FZ.x, DA.x * k.inv_sqrtK});
  flush_pair(v, deda, sb, PairAcc{FX.y, FY.y, FZ.y, DA.y * k.inv_sqrtK});
  flush_pair(v, deda, r0 + lane, PairAcc{-R.fx, -R.fy, -R.fz, R.da * k.inv_sqrtK});
}

// whether no pair of the tile may lie above the exp threshold, from its blocks' radii
// and largest Born radii
__device__ __forceinline__ bool blocks_far(const DevView& v, const GBConst& k, const Tile& T) {
  const float d = sqrtf(T.ox * T.ox + T.oy * T.oy + T.oz * T.oz) * 0.9999f - v.brad[T.bi] - v.brad[T.bj];
  return d > 0.f && d * d > k.sqrtK * v.bborn[T.bi] * 1.0001f * (k.sqrtK * v.bborn[T.bj]);
}

template <bool FAST, bool ENERGY>
__device__ __forceinline__ void gb_pair_single(const DevView& v, const GBConst& k, const Tile& T, int lane,
                                               const float* born, long long* deda, PairRows& rs,
                                               PairRowsE* re) {
  const bool full = tile_full(T);
  // the rarer passes: all-inside unmasked tiles have a body of their own (energies and
  // forces of 4,224 atoms without cutoff 85.5 -> 82.6 us), the masked bodies serve the rest
  if ((!FAST || ENERGY) && !(full && !tile_masked(T))) {
    if (full) gb_pair_tile<true, true, FAST, ENERGY>(v, k, T, lane, born, deda, rs, re);
    else gb_pair_tile<true, false, FAST, ENERGY>(v, k, T, lane, born, deda, rs, re);
  } else if (tile_masked(T)) {
    if (full) gb_pair_tile<true, true, FAST, ENERGY>(v, k, T, lane, born, deda, rs, re);
    else gb_pair_tile<true, false, FAST, ENERGY>(v, k, T, lane, born, deda, rs, re);
  } else {
    if (full) gb_pair_tile<false, true, FAST, ENERGY>(v, k, T, lane, born, deda, rs, re);
    else gb_pair_tile<false, false, FAST, ENERGY>(v, k, T, lane, born, deda, rs, re);
  }
}

// The force-only pass (every dynamics step).  FAST: of an all-inside tile pair only what
// the base law lacks, and nothing where no pair of it may lie above the exp threshold
// (most items of a large peptide): each lane asks that of one item of the warp's, by
// block bounds.  FAST off: calcBornForces (gbff.cpp:1189-1340), tile by tile; LJ and
// Coulomb come from the NB kernel with the GB object's own settings.
constexpr int kPairThreads = 128, kPairEThreads = 128;
template <bool FAST>
__global__ void __launch_bounds__(kPairThreads, 6) k_gb_pair(const __grid_constant__ DevView v, const __grid_constant__ GBConst k, const float* born, long long* deda) {
  pdl_sync();
  __shared__ PairRows rows[kPairThreads / 32];
  PairRows& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int ni = *v.nitems;
  for (long long first = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; first < ni; first += 32LL * nwarps) {
    const long long mine = first + (long long)lane * nwarps;
    bool work = mine < ni;
    if (FAST && work) {
      const int2 t = v.items[mine];
      if (t.y >= 0) {
        const Tile T = v.tiles[t.x], U = v.tiles[t.y];
        work = !(tile_full(T) && tile_full(U) && blocks_far(v, k, T) && blocks_far(v, k, U));
      }
    }
    for (unsigned m = __ballot_sync(0xffffffffu, work); m; m &= m - 1u) {
      const int2 t = v.items[first + (long long)(__ffs(m) - 1) * nwarps];
      const Tile T = v.tiles[t.x];
      if (t.y >= 0) {
        const Tile U = v.tiles[t.y];
        if (FAST && tile_full(T) && tile_full(U)) {
          gb_near_full2(v, k, T, U, lane, born, deda, rs);
          continue;
        }
        gb_pair_single<FAST, false>(v, k, U, lane, born, deda, rs, nullptr);
      }
      gb_pair_single<FAST, false>(v, k, T, lane, born, deda, rs, nullptr);
    }
  }
}

// the pass with energies, tile by tile
template <bool FAST>
__global__ void __launch_bounds__(kPairEThreads, 4) k_gb_pair_energy(const __grid_constant__ DevView v, const __grid_constant__ GBConst k, const float* born,
                                                                    long long* deda) {
  pdl_sync();
  __shared__ PairRowsE rows[kPairEThreads / 32];
  PairRowsE& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nt = *v.ntiles;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nwarps)
    gb_pair_single<FAST, true>(v, k, v.tiles[t], lane, born, deda, rs, &rs);
}

// self term, total dE/da and the chain-rule prefactor a^2/166 * dE/da * P4
__global__ void k_gb_self(DevView v, const double* charge, GBConst k, double premul, const long long* deda,
                          const double* born_d, float* chain, int energy) {
  pdl_sync();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  long long e = 0;
  if (s < v.nslots) {  // nslots is a multiple of 32: warps are whole
    const int a = v.sorted_atom[s];
    if (a < 0) {
      chain[s] = 0.f;
    } else {
      const double ai = born_d[a], q = charge[a];
      const double inv = 1.0 / ai;
      const double self = premul * q * q * inv;
      const double da = (double)deda[s] * (1.0 / kSumScale) - self * inv;
      chain[s] = (float)(ai * ai * (1.0 / 166.0) * da * (double)k.P4);
      if (energy) e = fix_energy_d(self);
    }
  }
  if (energy) {  // a warp's slots are one block of one system: one atomic per warp
    e = warp_sum_ll(e);
    if ((threadIdx.x & 31) == 0 && s < v.nslots)
      atomic_add_ll(&v.eacc[(size_t)v.slot_sys[s >> 5] * E_NSLOTS + E_POL_SELF], e);
  }
}

// ---------------------------------------------------------------------------
// pass 3: dE/da chain rule through the Born radii, both directions of a pair
// ---------------------------------------------------------------------------
__device__ __forceinline__ void flush_force(const DevView& v, int s, const PairAcc& a) { flush_pair(v, nullptr, s, a); }

// 0.25 (4 CCF - dCCF) of a pair in close contact, 1 otherwise
__device__ __forceinline__ float chain_fac(const GBConst& k, float r2, float rs) {
  const float rs2 = rs * rs;
  if (!gb_contact(k, r2, rs2)) return 1.f;
  float sn, cs;
  const float x = __fdividef(r2, rs2) * k.P5;
  sincospif(x, &sn, &cs);
  const float h = 0.5f - 0.5f * cs;
  return 0.25f * (4.f * h * h - 2.f * h * sn * (x * 3.14159265358979f));
}

// CTAs of 128 threads, six per SM (24 warps at 80 registers)
constexpr int kChainThreads = 128;
constexpr int kChainWarps = kChainThreads / 32;

// rows of the rotating block in the warp's shared memory, twice over (as BornRows)
struct ChainRows {
  float4 xy[64], zv[64];   // (x, x', y, y'), (z, z', V, V')
  float2 c[64], r[64];     // (c, c'), (R, R') (R for single tiles only)
};

// Born chain rule of a single tile, step-packed (as born_tile)
template <bool MASKED, bool FULL>
__device__ __forceinline__ void chain_tile(const DevView& v, const GBConst& k, const Tile& T, int lane, unsigned ex,
                                           const float* chain, ChainRows& rs) {
  const int si = T.bi * 32 + lane, j0 = T.bj * 32, l1 = (lane + 1) & 31;
  const float4 xi = v.xq[si], pi = v.par[si];
  {
    const float4 x0 = j_in_i_frame(v, T, lane), p0 = v.par[j0 + lane];
    const float c0 = -4.f * chain[j0 + lane];
    const float x1 = __shfl_sync(0xffffffffu, x0.x, l1), y1 = __shfl_sync(0xffffffffu, x0.y, l1);
    const float z1 = __shfl_sync(0xffffffffu, x0.z, l1), v1 = __shfl_sync(0xffffffffu, p0.w, l1);
    const float r1 = __shfl_sync(0xffffffffu, p0.z, l1), c1 = __shfl_sync(0xffffffffu, c0, l1);
    __syncwarp();
    rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x1, x0.y, y1);
    rs.zv[lane] = rs.zv[lane + 32] = make_float4(x0.z, z1, p0.w, v1);
    rs.c[lane] = rs.c[lane + 32] = make_float2(c0, c1);
    rs.r[lane] = rs.r[lane + 32] = make_float2(p0.z, r1);
    __syncwarp();
  }
  const float2 AX = f2(-xi.x), AY = f2(-xi.y), AZ = f2(-xi.z), RA = f2(pi.z), VA = f2(pi.w);
  const float2 CA = f2(-4.f * chain[si]);
  float2 FX = f2(0.f), FY = f2(0.f), FZ = f2(0.f);
  float2 FRX = f2(0.f), FRY = f2(0.f), FRZ = f2(0.f);   // minus the rotating atoms' sums
#pragma unroll 2
  for (int kk = 0; kk < 32; kk += 2) {
    const int j = lane + kk;
    const float4 P = rs.xy[j], Q = rs.zv[j];
    const float2 ax = __fadd2_rn(make_float2(P.x, P.y), AX), ay = __fadd2_rn(make_float2(P.z, P.w), AY);
    const float2 az = __fadd2_rn(make_float2(Q.x, Q.y), AZ);
    const float2 r2 = __ffma2_rn(az, az, __ffma2_rn(ay, ay, __fmul2_rn(ax, ax)));
    const float2 ir2 = make_float2(rcp_ftz(r2.x), rcp_ftz(r2.y));
    float2 w = __fmul2_rn(__ffma2_rn(CA, make_float2(Q.z, Q.w), __fmul2_rn(rs.c[j], VA)),
                          __fmul2_rn(__fmul2_rn(ir2, ir2), ir2));
    const float2 s = __fadd2_rn(rs.r[j], RA), lim = __fmul2_rn(__fmul2_rn(s, s), f2(k.invP5));
    if (__any_sync(0xffffffffu, r2.x <= lim.x || r2.y <= lim.y)) {
      w.x *= chain_fac(k, r2.x, s.x);
      w.y *= chain_fac(k, r2.y, s.y);
    }
    bool ia = still_in<FULL>(v, k, r2.x, si, j0 + (j & 31));
    bool ib = still_in<FULL>(v, k, r2.y, si, j0 + ((j + 1) & 31));
    if (MASKED) {
      ia = ia && !((ex >> kk) & 1u);
      ib = ib && !((ex >> kk) & 2u);
    }
    if (MASKED || !FULL) {
      w.x = ia ? w.x : 0.f;
      w.y = ib ? w.y : 0.f;
    }
    FX = __ffma2_rn(w, ax, FX); FY = __ffma2_rn(w, ay, FY); FZ = __ffma2_rn(w, az, FZ);
    FRX = __ffma2_rn(w, ax, FRX); FRY = __ffma2_rn(w, ay, FRY); FRZ = __ffma2_rn(w, az, FRZ);
    ROT2(FRX); ROT2(FRY); ROT2(FRZ);
  }
  const int lm = (lane + 31) & 31;
  const float frx = FRX.x + __shfl_sync(0xffffffffu, FRX.y, lm);
  const float fry = FRY.x + __shfl_sync(0xffffffffu, FRY.y, lm);
  const float frz = FRZ.x + __shfl_sync(0xffffffffu, FRZ.y, lm);
  flush_force(v, si, PairAcc{FX.x + FX.y, FY.x + FY.y, FZ.x + FZ.y, 0.f});
  flush_force(v, j0 + lane, PairAcc{-frx, -fry, -frz, 0.f});
}

// Born chain rule of an all-inside tile pair, step-packed: (c_i V_j + c_j V_i)
// (4 CCF - dCCF) / r^6 along d, with -4 folded into c (w then carries the held
// atom's sign and the factor 4 of the no-contact case); the CCF branch on the
// coarse-bound vote.
// FAR: no pair of the item in close contact.
template <bool FAR>
__device__ __forceinline__ void chain_loop2(const DevView& v, const GBConst& k, int lane, int r0, const ChainRows& rs,
                                            const float4& xa, const float4& xb, const float4& pa, const float4& pb,
                                            float ca, float cb, float c2, float2 FA[3], float2 FB[3], float2 FR[3]) {
  const float2 AX = f2(-xa.x), AY = f2(-xa.y), AZ = f2(-xa.z), BX = f2(-xb.x), BY = f2(-xb.y), BZ = f2(-xb.z);
  const float2 VA = f2(pa.w), VB = f2(pb.w), CA = f2(ca), CB = f2(cb);
  const float4 *xy = rs.xy + lane, *zv = rs.zv + lane;
  const float2* cr = rs.c + lane;
#pragma unroll 2
  for (int kk = 0; kk < 32; kk += 2) {
    const float4 P = xy[kk], Q = zv[kk];
    const float2 CR = cr[kk];
    const float2 X = make_float2(P.x, P.y), Y = make_float2(P.z, P.w), Z = make_float2(Q.x, Q.y);
    const float2 VR = make_float2(Q.z, Q.w);
    const float2 ax = __fadd2_rn(X, AX), ay = __fadd2_rn(Y, AY), az = __fadd2_rn(Z, AZ);
    const float2 bx = __fadd2_rn(X, BX), by = __fadd2_rn(Y, BY), bz = __fadd2_rn(Z, BZ);
    const float2 ra = __ffma2_rn(az, az, __ffma2_rn(ay, ay, __fmul2_rn(ax, ax)));
    const float2 rb = __ffma2_rn(bz, bz, __ffma2_rn(by, by, __fmul2_rn(bx, bx)));
    const float2 ia = make_float2(rcp_ftz(ra.x), rcp_ftz(ra.y));
    const float2 ib = make_float2(rcp_ftz(rb.x), rcp_ftz(rb.y));
    // -w of the plain law: (c_held V_rot + c_rot V_held) (-4) / r^6
    float2 wa = __fmul2_rn(__ffma2_rn(CA, VR, __fmul2_rn(CR, VA)), __fmul2_rn(__fmul2_rn(ia, ia), ia));
    float2 wb = __fmul2_rn(__ffma2_rn(CB, VR, __fmul2_rn(CR, VB)), __fmul2_rn(__fmul2_rn(ib, ib), ib));
    if (!FAR) {
      if (__any_sync(0xffffffffu, fminf(fminf(ra.x, ra.y), fminf(rb.x, rb.y)) <= c2)) {
        // rare: the rotating atoms' radii are read here, not staged
        const float R0 = v.par[r0 + ((lane + kk) & 31)].z, R1 = v.par[r0 + ((lane + kk + 1) & 31)].z;
        wa.x *= chain_fac(k, ra.x, pa.z + R0);
        wa.y *= chain_fac(k, ra.y, pa.z + R1);
        wb.x *= chain_fac(k, rb.x, pb.z + R0);
        wb.y *= chain_fac(k, rb.y, pb.z + R1);
      }
    }
    FA[0] = __ffma2_rn(wa, ax, FA[0]); FA[1] = __ffma2_rn(wa, ay, FA[1]); FA[2] = __ffma2_rn(wa, az, FA[2]);
    FB[0] = __ffma2_rn(wb, bx, FB[0]); FB[1] = __ffma2_rn(wb, by, FB[1]); FB[2] = __ffma2_rn(wb, bz, FB[2]);
    FR[0] = __ffma2_rn(wa, ax, __ffma2_rn(wb, bx, FR[0]));
    FR[1] = __ffma2_rn(wa, ay, __ffma2_rn(wb, by, FR[1]));
    FR[2] = __ffma2_rn(wa, az, __ffma2_rn(wb, bz, FR[2]));
    ROT2(FR[0]); ROT2(FR[1]); ROT2(FR[2]);
  }
}

__device__ __forceinline__ void chain_full2(const DevView& v, const GBConst& k, const Tile& A, const Tile& B, int lane,
                                            const float* chain, ChainRows& rs) {
  const int sa = A.bj * 32 + lane, sb = B.bj * 32 + lane, r0 = A.bi * 32;
  const int l1 = (lane + 1) & 31;
  const float4 xa = j_in_i_frame(v, A, lane), xb = j_in_i_frame(v, B, lane);
  const float4 pa = v.par[sa], pb = v.par[sb];
  const float ca = -4.f * chain[sa], cb = -4.f * chain[sb];
  float c2;
  bool far;
  {
    const float4 x0 = v.xq[r0 + lane], p0 = v.par[r0 + lane];
    const float c0 = -4.f * chain[r0 + lane];
    const float x1 = __shfl_sync(0xffffffffu, x0.x, l1), y1 = __shfl_sync(0xffffffffu, x0.y, l1);
    const float z1 = __shfl_sync(0xffffffffu, x0.z, l1), v1 = __shfl_sync(0xffffffffu, p0.w, l1);
    const float c1 = __shfl_sync(0xffffffffu, c0, l1);
    c2 = pair_contact2(k, make_float2(pa.z, pb.z), p0.z);
    far = item_far(xa, xb, x0, c2, c2);
    __syncwarp();
    rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x1, x0.y, y1);
    rs.zv[lane] = rs.zv[lane + 32] = make_float4(x0.z, z1, p0.w, v1);
    rs.c[lane] = rs.c[lane + 32] = make_float2(c0, c1);
    __syncwarp();
  }
  // (FR: minus the rotating atoms' sums)
  float2 FA[3], FB[3], FR[3];
#pragma unroll
  for (int c = 0; c < 3; c++) FA[c] = FB[c] = FR[c] = f2(0.f);
  if (far) chain_loop2<true>(v, k, lane, r0, rs, xa, xb, pa, pb, ca, cb, c2, FA, FB, FR);
  else chain_loop2<false>(v, k, lane, r0, rs, xa, xb, pa, pb, ca, cb, c2, FA, FB, FR);
  const int lm = (lane + 31) & 31;
  const float frx = FR[0].x + __shfl_sync(0xffffffffu, FR[0].y, lm);
  const float fry = FR[1].x + __shfl_sync(0xffffffffu, FR[1].y, lm);
  const float frz = FR[2].x + __shfl_sync(0xffffffffu, FR[2].y, lm);
  flush_force(v, sa, PairAcc{FA[0].x + FA[0].y, FA[1].x + FA[1].y, FA[2].x + FA[2].y, 0.f});
  flush_force(v, sb, PairAcc{FB[0].x + FB[0].y, FB[1].x + FB[1].y, FB[2].x + FB[2].y, 0.f});
  flush_force(v, r0 + lane, PairAcc{-frx, -fry, -frz, 0.f});
}

__device__ __forceinline__ void chain_single(const DevView& v, const GBConst& k, const Tile& T, int lane,
                                             const float* chain, ChainRows& rs) {
  const bool full = tile_full(T);
  if (tile_masked(T)) {
    unsigned ex, m14;
    tile_masks(v, T, lane, ex, m14);
    if (T.flags & 2) ex |= diag_exclusion(lane);
    if (full) chain_tile<true, true>(v, k, T, lane, ex, chain, rs);
    else chain_tile<true, false>(v, k, T, lane, ex, chain, rs);
  } else if (full) {
    chain_tile<false, true>(v, k, T, lane, 0u, chain, rs);
  } else {
    chain_tile<false, false>(v, k, T, lane, 0u, chain, rs);
  }
}

__global__ void __launch_bounds__(kChainThreads, 6) k_gb_chain(const __grid_constant__ DevView v, const __grid_constant__ GBConst k, const float* chain) {
  pdl_sync();
  __shared__ ChainRows rows[kChainWarps];
  ChainRows& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int ni = *v.nitems;
  for (int it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < ni; it += nwarps) {
    const int2 t = v.items[it];
    const Tile T = v.tiles[t.x];
    if (t.y >= 0) {
      const Tile U = v.tiles[t.y];
      if (tile_full(T) && tile_full(U)) {
        chain_full2(v, k, T, U, lane, chain, rs);
        continue;
      }
      chain_single(v, k, U, lane, chain, rs);
    }
    chain_single(v, k, T, lane, chain, rs);
  }
}

int tile_grid(Context& c) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
  long long want = (c.tile_cap + 7) / 8;
  long long g = (long long)sms * c.tile_ctas_per_sm;
  return (int)(want < g ? (want > 0 ? want : 1) : g);
}

int launch_gb(Context& c, const GBConst& k, double halfeconv, double born_offset, double premul, bool energy) {
  c.kernel_launches += 5;
  DevView v = c.view();
  cudaStream_t st = c.stream;
  int g = tile_grid(c);
  const Spread sp = spread(c.nslots);
  const int gp = g * (256 / kPairThreads), ge = g * (256 / kPairEThreads);
  if (k.fast && !energy && !c.gb_no_chain) launch_pdl(st, g * (256 / kBaseThreads), kBaseThreads, 0, k_gb_born<true>, v, k, c.d_gpol.p);
  else launch_pdl(st, g, kBornThreads, 0, k_gb_born<false>, v, k, c.d_gpol.p);
  launch_pdl(st, sp.grid, sp.threads, 0, k_gb_radii, v, c.d_gbT.p, c.d_gpol.p, born_sum_unit(c.gb), halfeconv, born_offset,
             c.d_born_f.p, c.d_born_d.p, c.d_bborn.p);
  if (c.gb_no_chain) {
    // a gradient call: energies (FP32 pair terms: they weight a loss), dE/da and the
    // pair terms' gradients in one pass, no forces
    const int e = launch_adj_gb_pair(c, k);
    if (e != PDGPU_OK) return e;
  } else if (energy) {
    if (!k.fast) launch_pdl(st, ge, kPairEThreads, 0, k_gb_pair_energy<false>, v, k, c.d_born_f.p, c.d_deda.p);
    else launch_pdl(st, ge, kPairEThreads, 0, k_gb_pair_energy<true>, v, k, c.d_born_f.p, c.d_deda.p);
  } else if (!k.fast) {
    launch_pdl(st, gp, kPairThreads, 0, k_gb_pair<false>, v, k, c.d_born_f.p, c.d_deda.p);
  } else {
    launch_pdl(st, 2 * gp, kPairThreads, 0, k_gb_pair<true>, v, k, c.d_born_f.p, c.d_deda.p);   // (unequal items: 222 -> 215 us)
  }
  launch_pdl(st, sp.grid, sp.threads, 0, k_gb_self, v, c.d_charge.p, k, premul, c.d_deda.p, c.d_born_d.p, c.d_chain_f.p,
                                energy ? 1 : 0);
  if (c.gb_no_chain || c.no_forces) c.kernel_launches -= 1;
  else launch_pdl(st, 2 * g, kChainThreads, 0, k_gb_chain, v, k, c.d_chain_f.p);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

// one GB pass on its own (timing probe): 1 Born sums, 2 fused pair (forces), 3 chain rule
int launch_gb_stage(Context& c, const GBConst& k, int stage) {
  DevView v = c.view();
  int g = tile_grid(c);
  c.kernel_launches += 1;
  if (stage == 1) launch_pdl(c.stream, g * (256 / kBaseThreads), kBaseThreads, 0, k_gb_born<true>, v, k, c.d_gpol.p);
  else if (stage == 2) launch_pdl(c.stream, 2 * g * (256 / kPairThreads), kPairThreads, 0, k_gb_pair<true>, v, k, c.d_born_f.p, c.d_deda.p);
  else launch_pdl(c.stream, 2 * g, kChainThreads, 0, k_gb_chain, v, k, c.d_chain_f.p);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

}  // namespace pdgpu
