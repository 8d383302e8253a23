// k_adjoint.cu — gradients of the nonbonded / GB energy with respect to the
// per-atom force-field parameters (charge, LJ radius, sqrt epsilon, GB radius,
// GB volume Vj, GB fixed term terms123).
//
// PD has no adjoint; its parameter derivatives are finite differences of
// Forcefield::calcEnergies after re-running setup() (nonbonded.cpp:1078-1084
// explains why setup must be repeated: calcCheckSum does not see parameter
// edits).  The energy being differentiated is PD's:
//   FF_NonBonded   nonbonded.cpp:687-833
//   GB (FastMode)  gbff.cpp:1546-1746 (pair + self terms), Born radii
//                  gbff.cpp:432-483 with a = -halfeconv / Gpol + BornRadiusOffset
// The derivative is the exact one of that energy (dE/dGpol = dE/da *
// halfeconv / Gpol^2), not PD's force-path shortcut a^2/166 (gbff.cpp:1790),
// which differs from it by the Born offset and by 166 vs halfeconv.
//
// Layout: the same tiles and slots as the force kernels.  Pair distances and
// most pair terms are FP32; for FF_NonBonded the Coulomb energy per unit charge
// product is formed in double-float (the force-switch form cancels badly in FP32).
// A charge gradient is a potential: a sum of many terms of both signs, which plain
// FP32 sums do not resolve to the 1e-4 a parameter fit checks against.  The
// kernels therefore sum per tile in compensated FP32 (value plus running
// rounding error, about 48 significant bits, on the FP32 pipe: GB300's FP64 rate
// is a small fraction of its FP32 rate), fed by every term of FF_NonBonded and by
// plain FP32 sums over 8 rotation steps of GB.  Per-tile sums enter 64-bit fixed
// point (2^32 per kcal/mol per parameter unit), so the result does not depend on
// scheduling.
#include "pdgpu_tile.cuh"

namespace pdgpu {

enum { G_Q = 0, G_R, G_EPS, G_GBR, G_VJ, G_NACC };

struct Acc3 {
  double a, b, c;
};

__device__ __forceinline__ long long fix_sum_d(double x) { return __double2ll_rn(x * kSumScale); }

// Compensated FP32 sum: hi carries the running sum and lo the rounding errors
// of its additions, each recovered exactly by Knuth's TwoSum (the _rn
// intrinsics keep the compiler from contracting or reordering the steps).
struct CSum {
  float hi, lo;
};

__device__ __forceinline__ void csum_add(CSum& c, float x) {
  const float s = __fadd_rn(c.hi, x);
  const float bb = __fsub_rn(s, c.hi);
  const float e = __fadd_rn(__fsub_rn(c.hi, __fsub_rn(s, bb)), __fsub_rn(x, bb));
  c.lo = __fadd_rn(c.lo, e);
  c.hi = s;
}

struct CAcc3 {
  CSum a, b, c;
};

__device__ __forceinline__ void acc_flush(const DevView& v, long long* g0, long long* g1, long long* g2, int s,
                                          const Acc3& x) {
  const double m = fabs(x.a) + fabs(x.b) + fabs(x.c);
  if (!(m < 1.0e9)) atomicOr(v.status, (unsigned)(m >= 1.0e9 ? ST_FIXED_OVERFLOW : ST_NAN));
  if (g0) atomic_add_ll(&g0[s], fix_sum_d(x.a));
  if (g1) atomic_add_ll(&g1[s], fix_sum_d(x.b));
  if (g2) atomic_add_ll(&g2[s], fix_sum_d(x.c));
}

// compensated sums into fixed point without FP64 work (fx32 holds below 2^29)
__device__ __forceinline__ void acc_flush(const DevView& v, long long* g0, long long* g1, long long* g2, int s,
                                          const CAcc3& x) {
  const float m = fabsf(x.a.hi) + fabsf(x.b.hi) + fabsf(x.c.hi);
  if (!(m < 2.6e8f)) {
    acc_flush(v, g0, g1, g2, s, Acc3{(double)x.a.hi + (double)x.a.lo, (double)x.b.hi + (double)x.b.lo,
                                     (double)x.c.hi + (double)x.c.lo});
    return;
  }
  if (g0) atomic_add_ll(&g0[s], fx32(x.a.hi) + fx32(x.a.lo));
  if (g1) atomic_add_ll(&g1[s], fx32(x.b.hi) + fx32(x.b.lo));
  if (g2) atomic_add_ll(&g2[s], fx32(x.c.hi) + fx32(x.c.lo));
}

// dE/dRmin of the LJ term eps (A - 2B) S(r), A = (R/r)^12, B = (R/r)^6, written
// without dividing by R (two zero-radius hydrogens give 0, not 0/0)
__device__ __forceinline__ float lj_dR(float R, float invr) {
  const float R2 = R * R, ir2 = invr * invr;
  const float b5 = R2 * R2 * R * (ir2 * ir2 * ir2);  // B / R
  const float t = R * invr, t2 = t * t;
  const float B = t2 * t2 * t2;
  return 12.f * b5 * (B - 1.f);                      // 12 (A - B) / R
}

// ---------------------------------------------------------------------------
// GB + vacuum pair terms in one pass over the tiles: energies, dE/da, dE/dq,
// dE/dRmin and dE/dsqrt(eps) (Born radii held fixed; their dependence on the GB
// parameters goes through dE/da in k_adj_born).  Step-packed as the GB force
// bodies (k_gb.cu): lane l holds i atom l, the j atoms l + kk and l + kk + 1 of
// the tile come as one FP32x2 pair from the warp's rows.  The gradient sums run
// over 8 rotation steps in FP32 (4 terms per half) and enter the compensated
// sums of the lane the atom lives in, so those never rotate.  Bound by FP32
// issue; 16 frames of 4,235 atoms: energies and gradients took 635 + 566 us in
// two passes of scalar bodies, 468 us in this one.
// ---------------------------------------------------------------------------
struct AdjRows {
  float4 xy[64], zq[64], se[64];   // step pairs (x, y), (z, q), (LJ radius, sqrt(eps)), twice over
  float2 a[64];                    // Born radii (pair pass), or w = dE/dGpol (Born pass)
};

// the sums of 8 steps: held atoms' into the lane's own, rotating atoms' into
// their home lane's (s: rotation steps made so far)
__device__ __forceinline__ void chunk_held(CSum& A, float2& c) {
  csum_add(A, c.x);
  csum_add(A, c.y);
  c = f2(0.f);
}
__device__ __forceinline__ void chunk_home(CSum& A, float2& c, int lane, int s) {
  csum_add(A, __shfl_sync(0xffffffffu, c.x, (lane - s) & 31));
  csum_add(A, __shfl_sync(0xffffffffu, c.y, (lane - s - 1) & 31));
  c = f2(0.f);
}

template <bool MASKED, bool FULL>
__device__ __forceinline__ void adj_gb_tile(const DevView& v, const GBConst& k, const Tile& T, int lane,
                                            const float4& xi, const float4& pi, float ai, unsigned ex, unsigned m14,
                                            unsigned dm, long long* deda, long long* gq, long long* gr, long long* ge,
                                            const AdjRows& rs) {
  const int si = T.bi * 32 + lane, j0 = T.bj * 32;
  const float2 X = f2(-xi.x), Y = f2(-xi.y), Z = f2(-xi.z), Q = f2(xi.w), R = f2(pi.x), E = f2(pi.y), AI = f2(ai);
  const float4 *xy = rs.xy + lane, *zq = rs.zq + lane, *se = rs.se + lane;
  const float2* aj = rs.a + lane;
  CAcc3 I = {}, J = {};
  float2 iq = f2(0.f), ir_ = f2(0.f), ie = f2(0.f), jq = f2(0.f), jr = f2(0.f), je = f2(0.f);
  float2 DA = f2(0.f), RA = f2(0.f), cv = f2(0.f), ce = f2(0.f), cp = f2(0.f);
  CSum ev = {0.f, 0.f}, ee = ev, ep_ = ev;
#pragma unroll 1
  for (int kk = 0; kk < 32; kk += 2) {
    const float4 P = xy[kk], ZQ = zq[kk], SE = se[kk];
    const float2 AJ = aj[kk];
    const float2 dx = __fadd2_rn(make_float2(P.x, P.y), X), dy = __fadd2_rn(make_float2(P.z, P.w), Y);
    const float2 dz = __fadd2_rn(make_float2(ZQ.x, ZQ.y), Z);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y)), ir2 = __fmul2_rn(ir, ir);
    bool ina = FULL || r2.x <= k.cut2, inb = FULL || r2.y <= k.cut2, xa = false, xb = false, ma = false, mb = false;
    if (MASKED) {
      ina = ina && !((dm >> kk) & 1u);
      inb = inb && !((dm >> kk) & 2u);
      xa = (ex >> kk) & 1u;
      xb = (ex >> kk) & 2u;
      ma = (m14 >> kk) & 1u;
      mb = (m14 >> kk) & 2u;
    }
    float2 S = f2(1.f), Sv = f2(1.f);
    if (!FULL) {
      const float2 r = __fmul2_rn(r2, ir);
      const float2 w = make_float2(fmaxf(r.x - k.inner, 0.f), fmaxf(r.y - k.inner, 0.f));
      const float2 sw = __ffma2_rn(__fmul2_rn(w, w), f2(-k.invw2), f2(1.f));
      S = __fmul2_rn(sw, sw);
      const float2 wv = make_float2(fmaxf(r.x - k.vdwinner, 0.f), fmaxf(r.y - k.vdwinner, 0.f));
      const float2 sv = __ffma2_rn(__fmul2_rn(wv, wv), f2(-k.vdwinvw2), f2(1.f));
      Sv = __fmul2_rn(sv, sv);
      Sv = make_float2(r.x < k.vdwcut ? Sv.x : 0.f, r.y < k.vdwcut ? Sv.y : 0.f);
    }
    // (selects, not products, below: the diagonal's own pair has r = 0)
    float2 el = __fmul2_rn(ir, S);   // Coulomb energy per unit q q, without its constant ec
    float2 ec = f2(k.econv_out);
    if (MASKED) el = __fmul2_rn(el, make_float2(ma ? k.elec14 : 1.f, mb ? k.elec14 : 1.f));
    // the GB term's code runs only when some lane may lie above the exp threshold
    // (warp vote, FP64 tie-break band included)
    const float2 aa = __fmul2_rn(AI, AJ);
    const float2 u = __fmul2_rn(__fmul2_rn(r2, f2(-0.25f)), make_float2(rcp_ftz(aa.x), rcp_ftz(aa.y)));
    const float lim = k.thresh - 4e-6f * fabsf(k.thresh);
    const bool na = ina && u.x >= lim, nb = inb && u.y >= lim;
    float2 po = f2(0.f);   // GB energy per unit q q
    float2 QQ = __fmul2_rn(Q, make_float2(ZQ.z, ZQ.w));
    if (__any_sync(0xffffffffu, na || nb)) {
      const float tie = 2e-6f * fabsf(k.thresh);
      bool ona = na && u.x > k.thresh, onb = nb && u.y > k.thresh;
      if (na && fabsf(u.x - k.thresh) <= tie) ona = gb_on_fp64(v, si, j0 + ((lane + kk) & 31), k.thresh_d);
      if (nb && fabsf(u.y - k.thresh) <= tie) onb = gb_on_fp64(v, si, j0 + ((lane + kk + 1) & 31), k.thresh_d);
      const float2 tg = make_float2(__expf(u.x), __expf(u.y));
      const float2 D = __ffma2_rn(tg, aa, r2);
      const float2 fgb = make_float2(rsqrtf(D.x), rsqrtf(D.y));
      float2 e = __fmul2_rn(__fmul2_rn(f2(k.premul), fgb), S);
      e = make_float2(ona ? e.x : 0.f, onb ? e.y : 0.f);
      po = __fadd2_rn(e, e);
      const float2 W = __fmul2_rn(__fmul2_rn(__fmul2_rn(__fmul2_rn(e, QQ), __fmul2_rn(fgb, fgb)), tg),
                                  __fadd2_rn(u, f2(-1.f)));
      DA = __ffma2_rn(W, AJ, DA);
      RA = __ffma2_rn(W, AI, RA);
      ec = make_float2(ona ? k.econv_in : k.econv_out, onb ? k.econv_in : k.econv_out);
    }
    el = __fmul2_rn(el, ec);
    if (MASKED || !FULL) el = make_float2(ina && !xa ? el.x : 0.f, inb && !xb ? el.y : 0.f);
    const float2 phi = __fadd2_rn(po, el);
    iq = __ffma2_rn(phi, make_float2(ZQ.z, ZQ.w), iq);
    jq = __ffma2_rn(phi, Q, jq);
    cp = __ffma2_rn(po, QQ, cp);
    ce = __ffma2_rn(el, QQ, ce);
    // LJ: e1 = A - 2B per unit sqrt(eps) sqrt(eps), and its derivative in R
    // (written without dividing by R: two zero-radius hydrogens give 0, not 0/0)
    const float2 RR = __fadd2_rn(R, make_float2(SE.x, SE.y)), R2 = __fmul2_rn(RR, RR);
    const float2 b5 = __fmul2_rn(__fmul2_rn(__fmul2_rn(R2, R2), RR), __fmul2_rn(__fmul2_rn(ir2, ir2), ir2));   // B / R
    const float2 B = __fmul2_rn(b5, RR);
    if (MASKED) Sv = __fmul2_rn(Sv, make_float2(ma ? k.vdw14 : 1.f, mb ? k.vdw14 : 1.f));
    float2 e1 = __fmul2_rn(__fmul2_rn(B, __fadd2_rn(B, f2(-2.f))), Sv);
    const float2 ee2 = __fmul2_rn(E, make_float2(SE.z, SE.w));
    float2 dR = __fmul2_rn(__fmul2_rn(__fmul2_rn(b5, __fadd2_rn(B, f2(-1.f))), f2(12.f)), __fmul2_rn(Sv, ee2));
    if (MASKED || !FULL) {
      e1 = make_float2(ina && !xa ? e1.x : 0.f, inb && !xb ? e1.y : 0.f);
      dR = make_float2(ina && !xa ? dR.x : 0.f, inb && !xb ? dR.y : 0.f);
    }
    ir_ = __fadd2_rn(ir_, dR);
    jr = __fadd2_rn(jr, dR);
    ie = __ffma2_rn(e1, make_float2(SE.z, SE.w), ie);
    je = __ffma2_rn(e1, E, je);
    cv = __ffma2_rn(e1, ee2, cv);
    ROT2(jq); ROT2(jr); ROT2(je); ROT2(RA);
    if ((kk & 6) == 6) {
      chunk_held(I.a, iq);
      chunk_held(I.b, ir_);
      chunk_held(I.c, ie);
      chunk_home(J.a, jq, lane, kk + 2);
      chunk_home(J.b, jr, lane, kk + 2);
      chunk_home(J.c, je, lane, kk + 2);
      chunk_held(ev, cv);
      chunk_held(ee, ce);
      chunk_held(ep_, cp);
    }
  }
  const float ra = RA.x + __shfl_sync(0xffffffffu, RA.y, (lane + 31) & 31), da = DA.x + DA.y;
  fix_range(v.status, fabsf(da) + fabsf(ra));
  atomic_add_ll(&deda[si], fx32(da));
  atomic_add_ll(&deda[j0 + lane], fx32(ra));
  acc_flush(v, gq, gr, ge, si, I);
  acc_flush(v, gq, gr, ge, j0 + lane, J);
  // the tile's energies meet over the warp in double-float and enter fixed point once
  const DF e0 = df_warp_sum(DF{ev.hi, ev.lo}), e1 = df_warp_sum(DF{ee.hi, ee.lo}), e2 = df_warp_sum(DF{ep_.hi, ep_.lo});
  const DF x = lane == 0 ? e0 : (lane == 1 ? e1 : e2);
  if (lane < 3) {
    long long* En = v.eacc + (size_t)v.slot_sys[T.bi] * E_NSLOTS;
    atomic_add_ll(&En[lane == 0 ? E_VDW : (lane == 1 ? E_ELEC : E_POL_CROSS)], fix_energy_d((double)x.h + (double)x.l));
  }
}

// the j block of a tile into the warp's rows (a0: the lane's value for rs.a)
__device__ __forceinline__ void adj_stage(const DevView& v, int lane, const float4& x0, const float4& p0, float s0,
                                          float e0, float a0, AdjRows& rs) {
  const int l1 = (lane + 1) & 31;
  const float x1 = __shfl_sync(0xffffffffu, x0.x, l1), y1 = __shfl_sync(0xffffffffu, x0.y, l1);
  const float z1 = __shfl_sync(0xffffffffu, x0.z, l1), q1 = __shfl_sync(0xffffffffu, x0.w, l1);
  const float s1 = __shfl_sync(0xffffffffu, s0, l1), e1 = __shfl_sync(0xffffffffu, e0, l1);
  const float a1 = __shfl_sync(0xffffffffu, a0, l1);
  __syncwarp();
  rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x1, x0.y, y1);
  rs.zq[lane] = rs.zq[lane + 32] = make_float4(x0.z, z1, x0.w, q1);
  rs.se[lane] = rs.se[lane + 32] = make_float4(s0, s1, e0, e1);
  rs.a[lane] = rs.a[lane + 32] = make_float2(a0, a1);
  __syncwarp();
}

constexpr int kAdjThreads = 128;
__global__ void __launch_bounds__(kAdjThreads, 4) k_adj_gb_pair(const __grid_constant__ DevView v, const __grid_constant__ GBConst k, const float* born, long long* deda, long long* gq,
                                                      long long* gr, long long* ge) {
  __shared__ AdjRows rows[kAdjThreads / 32];
  AdjRows& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nt = *v.ntiles;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nwarps) {
    const Tile T = v.tiles[t];
    const int si = T.bi * 32 + lane, sj = T.bj * 32 + lane;
    const float4 xi = v.xq[si], pi = v.par[si], xj = j_in_i_frame(v, T, lane), pj = v.par[sj];
    adj_stage(v, lane, xj, pj, pj.x, pj.y, born[sj], rs);
    const float ai = born[si];
    const bool full = tile_full_now(k, T, xi, xj);
    if (tile_masked(T)) {
      unsigned ex, m14;
      tile_masks(v, T, lane, ex, m14);
      const unsigned dm = (T.flags & 2) ? diag_exclusion(lane) : 0u;
      if (full) adj_gb_tile<true, true>(v, k, T, lane, xi, pi, ai, ex, m14, dm, deda, gq, gr, ge, rs);
      else adj_gb_tile<true, false>(v, k, T, lane, xi, pi, ai, ex, m14, dm, deda, gq, gr, ge, rs);
    } else {
      if (full) adj_gb_tile<false, true>(v, k, T, lane, xi, pi, ai, 0u, 0u, 0u, deda, gq, gr, ge, rs);
      else adj_gb_tile<false, false>(v, k, T, lane, xi, pi, ai, 0u, 0u, 0u, deda, gq, gr, ge, rs);
    }
  }
}

// the energy pass of a gradient call: energies and dE/da, and with them the pair
// terms' gradients into c.adj_g (G_NACC x nslots, cleared by the caller)
int launch_adj_gb_pair(Context& c, const GBConst& k) {
  const size_t ns = c.nslots;
  long long* g = c.adj_g;
  k_adj_gb_pair<<<2 * tile_grid(c), kAdjThreads, 0, c.stream>>>(c.view(), k, c.d_born_f.p, c.d_deda.p, g + G_Q * ns,
                                                                g + G_R * ns, g + G_EPS * ns);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Born-radius sums Gpol_i += P4 Vj CCF(r^2/(Ri+Rj)^2) / r^4 (bond order > 2,
// r <= GbsaStillCutoff): dE/dVj and dE/dR through w = dE/dGpol per slot.
// Step-packed; rows: (x, y), (z, P4 V), (R, -), w.  340 us on 16 frames of 4,235
// atoms as a scalar rotation, 210 us so.
// ---------------------------------------------------------------------------
// CCF, and dCCF/dx * dx/dR, of a pair (1 and 0 outside close contact)
__device__ __forceinline__ float2 ccf_grad(const GBConst& k, float r2, float rs) {
  const float rs2 = rs * rs;
  if (r2 > rs2 * k.invP5) return make_float2(1.f, 0.f);
  const float x = __fdividef(r2, rs2);
  float sn, cs;
  sincospif(x * k.P5, &sn, &cs);
  const float h = 0.5f - 0.5f * cs;
  return make_float2(h * h, h * sn * (k.P5 * 3.14159265358979f) * (-2.f * __fdividef(x, rs)));
}

template <bool MASKED, bool FULL>
__device__ __forceinline__ void adj_born_tile(const DevView& v, const GBConst& k, const Tile& T, int lane,
                                              const float4& xi, const float4& pi, float wi, unsigned ex,
                                              long long* gR, long long* gV, const AdjRows& rs) {
  const int si = T.bi * 32 + lane, j0 = T.bj * 32;
  const float2 X = f2(-xi.x), Y = f2(-xi.y), Z = f2(-xi.z), R = f2(pi.z), V = f2(pi.w), WI = f2(wi);
  const float4 *xy = rs.xy + lane, *zv = rs.zq + lane, *se = rs.se + lane;
  const float2* wj = rs.a + lane;
  CSum IV = {0.f, 0.f}, JV = IV, IR = IV, JR = IV;
  float2 iv = f2(0.f), jv = f2(0.f), irr = f2(0.f), jrr = f2(0.f);
  bool contact = false;   // some pair so far was in close contact (else the R sums stay zero)
#pragma unroll 1
  for (int kk = 0; kk < 32; kk += 2) {
    const float4 P = xy[kk], Q = zv[kk], SR = se[kk];
    const float2 WJ = wj[kk];
    const float2 dx = __fadd2_rn(make_float2(P.x, P.y), X), dy = __fadd2_rn(make_float2(P.z, P.w), Y);
    const float2 dz = __fadd2_rn(make_float2(Q.x, Q.y), Z);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    bool ina = true, inb = true;
    if (!FULL) {
      ina = r2.x <= k.still2;
      inb = r2.y <= k.still2;
      if (fabsf(r2.x - k.still2) <= 2e-6f * k.still2)
        ina = r2_slots_fp64(v, si, j0 + ((lane + kk) & 31)) <= k.still2_d;
      if (fabsf(r2.y - k.still2) <= 2e-6f * k.still2)
        inb = r2_slots_fp64(v, si, j0 + ((lane + kk + 1) & 31)) <= k.still2_d;
    }
    if (MASKED) {
      ina = ina && !((ex >> kk) & 1u);
      inb = inb && !((ex >> kk) & 2u);
    }
    const float2 i2 = make_float2(rcp_ftz(r2.x), rcp_ftz(r2.y));
    float2 h4 = __fmul2_rn(__fmul2_rn(i2, i2), f2(k.P4));
    if (MASKED || !FULL) h4 = make_float2(ina ? h4.x : 0.f, inb ? h4.y : 0.f);
    const float2 s = __fadd2_rn(R, make_float2(SR.x, SR.y));
    const float2 lim = __fmul2_rn(__fmul2_rn(s, s), f2(k.invP5));
    // close contact (r^2 <= rs^2 / P5, where the CCF switches on) is rare: its
    // branch runs on a warp vote
    if (__any_sync(0xffffffffu, (ina && r2.x <= lim.x) || (inb && r2.y <= lim.y))) {
      contact = true;
      const float2 ca = ccf_grad(k, r2.x, s.x), cb = ccf_grad(k, r2.y, s.y);
      const float2 gx = make_float2(ina ? ca.y : 0.f, inb ? cb.y : 0.f);
      const float2 gr = __fmul2_rn(__fmul2_rn(__ffma2_rn(WI, make_float2(Q.z, Q.w), __fmul2_rn(WJ, V)), h4), gx);
      irr = __fadd2_rn(irr, gr);
      jrr = __fadd2_rn(jrr, gr);
      h4 = __fmul2_rn(h4, make_float2(ina ? ca.x : 1.f, inb ? cb.x : 1.f));
    }
    iv = __ffma2_rn(WJ, h4, iv);   // dE/dV_i from Gpol_j
    jv = __ffma2_rn(WI, h4, jv);   // dE/dV_j from Gpol_i
    ROT2(jv);
    if (contact) { ROT2(jrr); }
    if ((kk & 6) == 6) {
      chunk_held(IV, iv);
      chunk_home(JV, jv, lane, kk + 2);
      if (contact) {
        chunk_held(IR, irr);
        chunk_home(JR, jrr, lane, kk + 2);
        contact = false;
      }
    }
  }
  acc_flush(v, gR, gV, nullptr, si, CAcc3{IR, IV, {0.f, 0.f}});
  acc_flush(v, gR, gV, nullptr, j0 + lane, CAcc3{JR, JV, {0.f, 0.f}});
}

__global__ void __launch_bounds__(kAdjThreads, 6) k_adj_born(const __grid_constant__ DevView v, const __grid_constant__ GBConst k, const float* w, long long* gR,
                                                   long long* gV) {
  __shared__ AdjRows rows[kAdjThreads / 32];
  AdjRows& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nt = *v.ntiles;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nwarps) {
    const Tile T = v.tiles[t];
    const int si = T.bi * 32 + lane, sj = T.bj * 32 + lane;
    const float4 xi = v.xq[si], pi = v.par[si], pj = v.par[sj];
    float4 xj = j_in_i_frame(v, T, lane);
    const bool full = tile_full_now(k, T, xi, xj);
    xj.w = pj.w;
    adj_stage(v, lane, xj, pj, pj.z, 0.f, w[sj], rs);
    const float wi = w[si];
    if (tile_masked(T)) {
      unsigned ex, m14;
      tile_masks(v, T, lane, ex, m14);
      if (T.flags & 2) ex |= diag_exclusion(lane);
      if (full) adj_born_tile<true, true>(v, k, T, lane, xi, pi, wi, ex, gR, gV, rs);
      else adj_born_tile<true, false>(v, k, T, lane, xi, pi, wi, ex, gR, gV, rs);
    } else {
      if (full) adj_born_tile<false, true>(v, k, T, lane, xi, pi, wi, 0u, gR, gV, rs);
      else adj_born_tile<false, false>(v, k, T, lane, xi, pi, wi, 0u, gR, gV, rs);
    }
  }
}

// dE/dGpol per slot: (dE/da from the pair pass - E_self / a) * halfeconv / Gpol^2
__device__ __forceinline__ double dE_dGpol(const DevView& v, const double* terms123, const long long* gpol,
                                           const long long* deda, double gscale, double premul, double halfeconv,
                                           int s, int a) {
  const double G = terms123[a] + (double)gpol[s] * gscale;
  const double ai = v.born[a], q = v.charge[a];
  const double da = (double)deda[s] * (1.0 / kSumScale) - premul * q * q / (ai * ai);
  return da * halfeconv / (G * G);
}

__global__ void k_adj_w(DevView v, const double* terms123, const long long* gpol, const long long* deda,
                        double gscale, double premul, double halfeconv, float* w) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= v.nslots) return;
  int a = v.sorted_atom[s];
  w[s] = a < 0 ? 0.f : (float)dE_dGpol(v, terms123, gpol, deda, gscale, premul, halfeconv, s, a);
}

// ---------------------------------------------------------------------------
// NB (FF_NonBonded) pair terms: dE/dq, dE/dRmin, dE/dsqrt(eps).  The Coulomb
// energy per unit charge product is formed in double-float from the FP32 distance
// and its sums are double-float; the LJ terms are FP32, each entered into a
// compensated sum.  (In FP64, with FP64 sums on the rotation, the pass took
// 751 us on 4 frames of 1,094 waters, bound by the FP64 pipe; 120 us so.)
// ---------------------------------------------------------------------------
// Coulomb energy of a pair per unit q q econv (elec14 aside): nb_pair's law
template <int ELEC>
__device__ __forceinline__ DF nb_phi_df(const NBEConst& e, float r2f) {
  const DF r2 = DF{r2f, 0.f}, ir = df_rsqrt(r2);
  if (ELEC == 1) return ir;
  const DF r = df_norm(df_mul(r2, ir));
  const DF w = df_norm(df_sub(r, e.inner));
  if (ELEC == 3) {
    if (w.h <= 0.f) return ir;
    const DF s = df_norm(df_sub(DF{1.f, 0.f}, df_mul(w, df_norm(df_mul(w, e.invw2)))));
    return df_norm(df_mul(ir, df_norm(df_mul(s, s))));
  }
  // Steinbach & Brooks force switch, nonbonded.cpp:798-819
  if (w.h <= 0.f) return df_norm(df_sub(ir, e.eshift));
  const DF c = df_norm(df_sub(e.cut, r));
  DF h = df_norm(df_add(e.q2, df_mul(e.q3, r)));
  h = df_norm(df_add(e.q1, df_mul(h, r)));
  h = df_norm(df_add(e.q0, df_mul(h, r)));
  h = df_norm(df_mul(df_norm(df_mul(h, ir)), df_norm(df_mul(df_norm(df_mul(c, c)), c))));
  return df_norm(df_mul(e.sA, h));
}

template <int ELEC, bool MASKED>
__device__ __forceinline__ void adj_nb_tile(const DevView& v, const NBConst& k, const Tile& T, const NBEConst& e,
                                            const SystemInfo& S, int lane, int si, const float4& xi, const float4& pi,
                                            unsigned ex, unsigned m14, CAcc3& I, CAcc3& J) {
  float4 xj = v.xq[T.bj * 32 + lane];
  float4 pj = v.par[T.bj * 32 + lane];
  float Lx = 1.f, Ly = 1.f, Lz = 1.f;
  if (S.periodic) {
    Lx = (float)S.box[0]; Ly = (float)S.box[1]; Lz = (float)S.box[2];
  }
  xj.x += T.ox;
  xj.y += T.oy;
  xj.z += T.oz;
  const bool mi = T.flags & 1;
  const float iLx = 1.f / Lx, iLy = 1.f / Ly, iLz = 1.f / Lz;
#pragma unroll 2
  for (int kk = 0; kk < 32; kk++) {
    float dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
    if (mi) {
      dx -= Lx * rintf(dx * iLx);
      dy -= Ly * rintf(dy * iLy);
      dz -= Lz * rintf(dz * iLz);
    }
    float r2 = dx * dx + dy * dy + dz * dz;
    bool listed = true;
    if (MASKED) listed = !((ex >> kk) & 1u);
    bool in = r2 <= k.cut2;
    if (listed && (fabsf(r2 - k.cut2) <= 2e-6f * k.cut2 || fabsf(r2 - k.vdwcut2) <= 2e-6f * k.vdwcut2)) {
      const double r2d = r2_fp64(v, S, si, T.bj * 32 + ((lane + kk) & 31));
      in = r2d <= k.cut2_dd;
      r2 = (float)r2d;
    }
    if (listed && in) {
      const bool is14 = MASKED && ((m14 >> kk) & 1u);
      const float sv = is14 ? k.vdw14 : 1.f;
      if (ELEC != 0) {
        DF phi = df_norm(df_mul(nb_phi_df<ELEC>(e, r2), e.econv));
        if (is14) phi = df_norm(df_mul(phi, e.elec14));
        const DF a = df_norm(df_scale(phi, xj.w)), b = df_norm(df_scale(phi, xi.w));
        csum_add(I.a, a.h);
        I.a.lo = __fadd_rn(I.a.lo, a.l);
        csum_add(J.a, b.h);
        J.a.lo = __fadd_rn(J.a.lo, b.l);
      }
      const float invr = rsqrtf(r2), r = r2 * invr;
      if (k.dovdw && r < (float)k.vdwcut_d) {
        float Sv = sv;
        if (r > (float)k.vdwinner_d) {
          const float u = r - (float)k.vdwinner_d;
          const float sw = 1.f - u * u * (float)k.vdwinvw2_d;
          Sv *= sw * sw;
        }
        const float R = pi.x + pj.x, t2 = R * R * invr * invr, B = t2 * t2 * t2;
        const float dR = lj_dR(R, invr) * Sv * pi.y * pj.y;
        const float e1 = (B * B - 2.f * B) * Sv;   // energy per unit sqrt(eps_i) sqrt(eps_j)
        csum_add(I.b, dR);
        csum_add(J.b, dR);
        csum_add(I.c, e1 * pj.y);
        csum_add(J.c, e1 * pi.y);
      }
    }
    ROT(xj.x); ROT(xj.y); ROT(xj.z); ROT(xj.w); ROT(pj.x); ROT(pj.y);
    ROT(J.a.hi); ROT(J.a.lo); ROT(J.b.hi); ROT(J.b.lo); ROT(J.c.hi); ROT(J.c.lo);
  }
}

template <int ELEC>
__global__ void __launch_bounds__(256) k_adj_nb(const __grid_constant__ DevView v, const __grid_constant__ NBConst k, const __grid_constant__ NBEConst e, long long* gq, long long* gr, long long* ge) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nt = *v.ntiles;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nwarps) {
    const Tile T = v.tiles[t];
    const int si = T.bi * 32 + lane;
    const float4 xi = v.xq[si], pi = v.par[si];
    const SystemInfo& S = v.sys[v.slot_sys[T.bi]];
    unsigned ex = 0u, m14 = 0u;
    if (T.mask >= 0) {
      uint2 m = v.masks[T.mask * 32 + lane];
      ex = m.x;
      m14 = m.y;
    }
    if (T.flags & 2) ex |= diag_exclusion(lane);
    CAcc3 I = {}, J = {};
    if (tile_masked(T)) adj_nb_tile<ELEC, true>(v, k, T, e, S, lane, si, xi, pi, ex, m14, I, J);
    else adj_nb_tile<ELEC, false>(v, k, T, e, S, lane, si, xi, pi, ex, m14, I, J);
    acc_flush(v, gq, gr, ge, si, I);
    acc_flush(v, gq, gr, ge, T.bj * 32 + lane, J);
  }
}

// ---------------------------------------------------------------------------
// fixed point per slot -> J per parameter unit, original atom order
// ---------------------------------------------------------------------------
struct AdjOut {
  double *q, *r, *e, *R, *V, *T;
};

__global__ void k_adj_out(DevView v, const long long* g, int nslots, bool gb, const double* terms123,
                          const long long* gpol, const long long* deda, double gscale, double premul,
                          double halfeconv, double eps_unit, AdjOut o) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= v.nslots) return;
  int a = v.sorted_atom[s];
  if (a < 0) return;
  const double f = 1.0 / kSumScale;
  double gq = (double)g[G_Q * (size_t)nslots + s] * f;
  if (gb) {
    const double ai = v.born[a];
    gq += 2.0 * premul * v.charge[a] / ai;  // self energy premul q^2 / a
  }
  if (o.q) o.q[a] = gq * kKcalMolToJ;
  if (o.r) o.r[a] = (double)g[G_R * (size_t)nslots + s] * f * kKcalMolToJ;
  if (o.e) o.e[a] = (double)g[G_EPS * (size_t)nslots + s] * f * eps_unit * kKcalMolToJ;
  if (o.R) o.R[a] = gb ? (double)g[G_GBR * (size_t)nslots + s] * f * kKcalMolToJ : 0.0;
  if (o.V) o.V[a] = gb ? (double)g[G_VJ * (size_t)nslots + s] * f * kKcalMolToJ : 0.0;
  if (o.T) o.T[a] = gb ? dE_dGpol(v, terms123, gpol, deda, gscale, premul, halfeconv, s, a) * kKcalMolToJ : 0.0;
}


// Runs after the energy pass of the same component (its Born radii, Gpol sums,
// dE/da and, for GB, the pair terms' gradients are there already).  g: G_NACC *
// nslots fixed-point accumulators, cleared before that pass; w: nslots floats
// (written in full here).
int launch_adjoint(Context& c, unsigned what, const AdjScratch& a, double* d_q, double* d_r, double* d_e, double* d_R,
                   double* d_V, double* d_T) {
  DevView v = c.view();
  cudaStream_t st = c.stream;
  const int ns = c.nslots;
  const int grid = tile_grid(c), nb = (ns + 255) / 256;
  const bool gb = (what & PDGPU_GB) != 0;
  const double ec = econv_kcal();
  const double halfeconv = 0.5 * ec;
  const double premul = gb ? -0.5 * ec * (1.0 / c.gb.DielectricSolute - 1.0 / c.gb.DielectricSolvent) : 0.0;
  const double gscale = gb ? born_sum_unit(c.gb) : 0.0;
  long long* g = a.g;
  if (gb) {
    GBConst k = make_gb_const(c.gb, c.list_radius_built);
    c.kernel_launches += 2;
    k_adj_w<<<nb, 256, 0, st>>>(v, c.d_gbT.p, c.d_gpol.p, c.d_deda.p, gscale, premul, halfeconv, a.w);
    k_adj_born<<<2 * grid, kAdjThreads, 0, st>>>(v, k, a.w, g + G_GBR * (size_t)ns, g + G_VJ * (size_t)ns);
  } else {
    long long *gq = g + G_Q * (size_t)ns, *gr = g + G_R * (size_t)ns, *ge = g + G_EPS * (size_t)ns;
    const NBConst k = make_nb_const(c.nb);
    const NBEConst e = make_nbe_const(k);
    c.kernel_launches += 1;
    switch (k.elecmode) {
      case 0: k_adj_nb<0><<<grid, 256, 0, st>>>(v, k, e, gq, gr, ge); break;
      case 1: k_adj_nb<1><<<grid, 256, 0, st>>>(v, k, e, gq, gr, ge); break;
      case 3: k_adj_nb<3><<<grid, 256, 0, st>>>(v, k, e, gq, gr, ge); break;
      default: k_adj_nb<4><<<grid, 256, 0, st>>>(v, k, e, gq, gr, ge); break;
    }
  }
  AdjOut o = {d_q, d_r, d_e, d_R, d_V, d_T};
  c.kernel_launches += 1;
  k_adj_out<<<nb, 256, 0, st>>>(v, g, ns, gb, c.d_gbT.p, c.d_gpol.p, c.d_deda.p, gscale, premul, halfeconv,
                                std::sqrt(kNa / kKcal2J), o);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

int clear_adjoint(Context& c, const AdjScratch& a) {
  return cudaMemsetAsync(a.g, 0, sizeof(long long) * G_NACC * (size_t)c.nslots, c.stream) == cudaSuccess
             ? PDGPU_OK
             : PDGPU_ERR_CUDA;
}

// the context's own scratch, allocated on first use
int adjoint_scratch(Context& c, AdjScratch& a) {
  if (c.d_adj.n < (size_t)G_NACC * c.nslots) {
    if (c.d_adj.alloc((size_t)G_NACC * c.nslots) != cudaSuccess) return PDGPU_ERR_CUDA;
    if (c.d_adj_w.alloc((size_t)c.nslots) != cudaSuccess) return PDGPU_ERR_CUDA;
  }
  a = AdjScratch{c.d_adj.p, c.d_adj_w.p};
  return PDGPU_OK;
}

// ---------------------------------------------------------------------------
// Fixed scratch for the gradient call of hosts that must not allocate device
// memory inside a call.  cudaMalloc and cudaFree synchronise the whole device,
// so a host that keeps other streams busy (a fitting loop beside dynamics of
// other replicas), or whose own pool allocator holds the free memory, cannot
// let pdgpu_param_grad_device allocate its scratch on first use.  This array
// sits in the library's static device data instead: kNoAllocMaxSlots sorted
// slots, G_NACC int64 accumulators and one float each (2.75 MiB), held by every
// GPU that loads the library until the process exits.  All contexts on a
// device share it, so calls whose GPU work overlaps race.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_adj_scratch[(size_t)kNoAllocMaxSlots *
                                                             (G_NACC * sizeof(long long) + sizeof(float))];

int adjoint_scratch_static(Context& c, AdjScratch& a) {
  if (c.nslots > kNoAllocMaxSlots) return PDGPU_ERR_CAPACITY;
  // The array's device address on the current device (the caller made the
  // context's device current).  In host code the array's name only stands in
  // for the symbol.  Looked up on every call: the lookup is cheap once the
  // module is loaded, keeps no host-side cache (nothing to go stale after a
  // device reset, nothing shared between host threads), and the first call on
  // a device may load the library's device code there.
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_adj_scratch) != cudaSuccess || !p) return PDGPU_ERR_CUDA;
  unsigned char* base = static_cast<unsigned char*>(p);
  a.g = reinterpret_cast<long long*>(base);
  a.w = reinterpret_cast<float*>(base + (size_t)kNoAllocMaxSlots * G_NACC * sizeof(long long));
  return PDGPU_OK;
}

}  // namespace pdgpu
