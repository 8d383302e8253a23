// k_nb.cu — LJ + Coulomb tile kernel (FF_NonBonded) and force finalisation.
//
// Pair law: PD src/mmlib/forcefields/nonbonded.cpp:687-833
//   (T_fast2 instantiation with VdwMode = EnergySwitch and ElecMode picked by
//    the dispatch at nonbonded.cpp:1222-1246).
// Every listed pair j < i inside Cutoff contributes once; bond order <= 2
// pairs are zero, 1-4 pairs are scaled by Vdw14Scaling / Elec14Scaling.
#include <algorithm>

#include "pdgpu_tile.cuh"

namespace pdgpu {

// the pair decision for pairs whose FP32 distance lies at a hard cutoff
__device__ __noinline__ double nb_r2_fp64(const DevView& v, const SystemInfo& S, int sa, int sb) {
  return r2_fp64(v, S, sa, sb);
}

struct NBAcc {
  float fx, fy, fz;
};

// Force part of the pair law in FP32: dE/dr divided by r.
template <int ELEC>
__device__ __forceinline__ float nb_force_f(const NBConst& k, float r2, float rsum, float eps, float qq) {
  const float invr = rsqrtf(r2), ir2 = invr * invr;
  const float r = r2 * invr;
  float g = 0.f;
  // switching without a branch: below the inner cutoff u = 0, so sw = 1 and the
  // derivative term is exactly 0 (same value as the unswitched law); a branch
  // here splits warps across the switching shell, which holds ~40% of the pairs
  if (k.dovdw) {
    const float t2 = rsum * rsum * ir2;
    const float B = t2 * t2 * t2, A = B * B;
    const float gv = -12.f * eps * ir2 * (A - B);
    const float u = fmaxf(r - k.vdwinner_f, 0.f);
    const float sw = 1.f - u * u * k.vdwinvw2_f;
    const float gs = sw * sw * gv + eps * (A - 2.f * B) * (-4.f * k.vdwinvw2_f * u * sw) * invr;
    g += r < k.vdwcut_f ? gs : 0.f;
  }
  if (ELEC == 1) {
    g -= qq * invr * ir2;
  } else if (ELEC == 3) {
    const float Ee = qq * invr;
    const float ge = -Ee * ir2;
    const float u = fmaxf(r - k.inner_f, 0.f);
    const float sw = 1.f - u * u * k.invw2_f;
    g += sw * sw * ge + Ee * (-4.f * k.invw2_f * u * sw) * invr;
  } else if (ELEC == 4) {
    // Steinbach & Brooks force switch, nonbonded.cpp:798-819
    if (r > k.inner_f) {
      const float c2mr2 = k.cut2 - r2;
      g -= qq * k.sA_f * ir2 * c2mr2 * c2mr2 * (k.fsw_k + 2.f * r2) * invr;
    } else {
      g -= qq * ir2 * invr;
    }
  }
  return g;
}

// 32 rotation steps of one work item: lane i holds an i atom, (xj, pj) the
// lane's j atom already in i's frame.  Tiles: j slot jb + lane, per-pair image
// when mi.  GROUP: the j atoms of a group (slots in gent[].w, -1 = empty lane,
// parked far away), never masked, one image.
template <int ELEC, bool MASKED, bool GROUP>
__device__ __forceinline__ void nb_rot(const DevView& v, const NBConst& k, const SystemInfo& S, int lane, int si,
                                      const float4& xi, const float4& pi, float qi, unsigned ex, unsigned m14,
                                      float4 xj, float4 pj, bool mi_tile, int jb, const float4* gent, NBAcc& I,
                                      NBAcc& J) {
  const bool mi = !GROUP && mi_tile;
  float Lx = 1.f, Ly = 1.f, Lz = 1.f;
  if (!GROUP && S.periodic) {
    Lx = (float)S.box[0]; Ly = (float)S.box[1]; Lz = (float)S.box[2];
  }
  const float iLx = 1.f / Lx, iLy = 1.f / Ly, iLz = 1.f / Lz;
#pragma unroll 4
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
    if (listed && (fabsf(r2 - k.cut2) <= 2e-6f * k.cut2 ||
                   fabsf(r2 - k.vdwcut2) <= 2e-6f * k.vdwcut2)) {
      // at a hard cutoff: decide, and take the distance, in FP64 (FP64 work only on this branch)
      const int sjr = GROUP ? __float_as_int(gent[(lane + kk) & 31].w) : jb + ((lane + kk) & 31);
      const double d2 = nb_r2_fp64(v, S, si, sjr);
      in = d2 <= k.cut2_dd;
      r2 = (float)d2;
    }
    if (listed && in) {
      const bool is14 = MASKED && ((m14 >> kk) & 1u);
      const float eps = pi.y * pj.y * (is14 ? k.vdw14 : 1.f);
      const float qq = qi * xj.w * (is14 ? k.elec14 : 1.f);
      const float fs = nb_force_f<ELEC>(k, r2, pi.x + pj.x, eps, qq);
      I.fx += fs * dx; I.fy += fs * dy; I.fz += fs * dz;
      J.fx -= fs * dx; J.fy -= fs * dy; J.fz -= fs * dz;
    }
    // rotate the j atom (data + its force accumulator) one lane down
    const int src = (lane + 1) & 31;
    xj.x = __shfl_sync(0xffffffffu, xj.x, src);
    xj.y = __shfl_sync(0xffffffffu, xj.y, src);
    xj.z = __shfl_sync(0xffffffffu, xj.z, src);
    xj.w = __shfl_sync(0xffffffffu, xj.w, src);
    pj.x = __shfl_sync(0xffffffffu, pj.x, src);
    pj.y = __shfl_sync(0xffffffffu, pj.y, src);
    J.fx = __shfl_sync(0xffffffffu, J.fx, src);
    J.fy = __shfl_sync(0xffffffffu, J.fy, src);
    J.fz = __shfl_sync(0xffffffffu, J.fz, src);
  }
}

// ---------------------------------------------------------------------------
// Pair energies.  FP32 cannot hold them (water's electrostatics cancel ~5000
// fold, and so do the force-switch polynomials), and the FP64 pipe is narrow:
// they are formed in double-float arithmetic (pdgpu_df.cuh, ~45 bits) from
// positions and parameters held as double-floats, in a pass of their own beside
// the force pass.  It lists the pairs inside the cutoff, with the force pass's
// items and skipping and nothing else in the loop, and deals the list over the
// lanes, so the ~300 instructions of a pair's energy run on full warps; an item
// passes its odd pairs on from one eighth to the next.  Against 64-bit sums the
// energies are within 3e-8 kcal/mol on up to 89,956 atoms (one fixed-point rounding per
// item); the same pass with constants short of 64 bits left 1.2e-7, and 1.3e-4 in virials.
// Bound by the FMA pipe and, in small systems, by the latency of its chains: two pairs
// a lane in packed arithmetic.  FP64 pair energies on the rotation, with the forces:
// 5.85 ms on the solvated 22,489 atoms at 15 A (force switch), 0.331 ms on 667 waters
// at 12 A; scalar double-float on a list kept by the force rotation: 0.461 and 0.046
// ms, 0.119 ms on 4,235 atoms without cutoff; this pass 0.366, 0.032 and 0.105 ms beside
// force passes of 0.060, 0.009 and 0.019 ms (left out of calls that read no forces).
// ---------------------------------------------------------------------------

// remainders of the packed slots (before each energy pass)
__global__ void k_df_records(DevView v, const double* charge, float4* rlo, float2* plo) {
  pdl_sync();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= v.nslots) return;
  const int a = v.sorted_atom[s];
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 p = make_float2(0.f, 0.f);
  if (a >= 0) {
    const int b = s >> 5;
    const SystemInfo& S = v.sys[v.slot_sys[b]];
    const float4 x = v.xq[s], q = v.par[s];
    const float h[3] = {x.x, x.y, x.z};
    float l[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double d = v.pos[3 * a + c] - v.center[3 * b + c];
      if (S.periodic) d -= S.box[c] * rint(d * S.ibox[c]);
      l[c] = (float)(d - (double)h[c]);
    }
    r = make_float4(l[0], l[1], l[2], (float)(charge[a] - (double)x.w));
    p = make_float2((float)(v.radius[a] - (double)q.x), (float)(v.sqeps[a] - (double)q.y));
  }
  rlo[s] = r;
  plo[s] = p;
}

struct NBESum {
  DF2 vdw, elec, vir;
  float2 f;   // of the pairs' force magnitudes: range check
};

// what an item keeps in shared memory: its atoms as double-floats in the i
// block's frame (a tile's j block, or two groups) and the list of pairs
constexpr int kNbList = 512 + 64;
struct NBEShared {
  float4 ih[32], il[32], ip[32];   // (x, y, z, q) high and low parts; (R, sqrt(eps)) high and low
  float4 jh[64], jl[64], jp[64];
  int js[64];                      // j slots
  unsigned short pair[2][kNbList]; // a warp's list: i row | j row << 5 | 1-4 << 11
  DF sum[3];                       // the second warp's sums
};

// r less an inner radius, normalised: the sign of a difference below one unit of r.h is
// in the low part (a virial off by 3e-5 where it was not looked at), and the radius's
// rest counts
__device__ __forceinline__ DF2 nb_beyond(DF2 r, DF inner, float rest) {
  DF2 w = df_norm(df_sub(r, df2(inner)));
  w.l = __fadd2_rn(w.l, f2(-rest));
  return w;
}

// S = (1 - w^2 / width^2)^2 and r S' of an energy switch, w = r - inner > 0 for one of
// the two pairs at least; 1 and 0 for a pair inside
__device__ __forceinline__ void nb_switch_df(DF2 r, DF2 w, DF invw2, DF2& S, DF2& dS) {
  w = df_select(w.h.x > 0.f, w.h.y > 0.f, w, df2(DF{0.f, 0.f}));
  const DF2 wi = df_mul(w, df2(invw2));
  const DF2 sw = df_norm(df_sub(df2(DF{1.f, 0.f}), df_mul(w, wi)));
  S = df_norm(df_sqr(sw));
  dS = df_norm(df_scale2(df_mul(df_mul(wi, sw), r), -4.f));
}

// a per-pair-image tile's box; minus the images to take off a displacement
struct NBEBox {
  bool mi;
  DF x, y, z;
  float ix, iy, iz, tx, ty, tz;
};
__device__ __forceinline__ float2 nb_images(float2 d, float iL) {
  constexpr float kRint = 12582912.f;   // 1.5 2^23: adding and taking it off rounds to an integer
  return __fadd2_rn(__ffma2_rn(d, f2(-iL), f2(kRint)), f2(-kRint));
}

// A pair whose terms exceed kNbLarge (atoms nearly on one another): 2^-45 of them is
// beyond the fixed point's resolution, in its sums too, so it goes in FP64 straight into
// these.
constexpr float kNbLarge = 4096.f;   // kcal/mol: 2^-44 of it is 2^-32
template <int ELEC>
__device__ __noinline__ void nb_energy_large(const DevView& v, const NBConst& k, const SystemInfo& S, int si, int sj,
                                             bool is14) {
  const int a = v.sorted_atom[si], b = v.sorted_atom[sj];
  if (a < 0 || b < 0) return;
  const double eps = v.sqeps[a] * v.sqeps[b] * (is14 ? k.vdw14_d : 1.0);
  const double qq = v.charge[a] * v.charge[b] * k.econv_diel_d * (is14 ? k.elec14_d : 1.0);
  double ev = 0.0, ee = 0.0, vir;
  nb_pair<ELEC>(k, nb_r2_fp64(v, S, si, sj), v.radius[a] + v.radius[b], eps, qq, ev, ee, vir);
  long long* E = v.eacc + (size_t)v.slot_sys[si >> 5] * E_NSLOTS;
  atomic_add_ll(&E[E_VDW], fix_energy_d(ev));
  atomic_add_ll(&E[E_ELEC], fix_energy_d(ee));
  atomic_add_ll(&E[E_VIRIAL], fix_energy_d(vir));
}

// energies of two listed pairs into the sums (same law as the force bodies; pair b
// counts only if two).  Products of products stay unnormalised where their l holds a
// few roundings of h: what df_mul leaves out is then below 1e-13, of either sign.
template <int ELEC, bool SW>
__device__ __forceinline__ void nb_energy_df2(const DevView& v, const NBConst& k, const NBEConst& e,
                                              const SystemInfo& S, const NBEBox& box, int ibase, const NBEShared* sh,
                                              unsigned ca, unsigned cb, bool two, NBESum& sum) {
  const int ia = ca & 31, ib = cb & 31, ja = (ca >> 5) & 63, jb = (cb >> 5) & 63;
  const float4 xha = sh->ih[ia], xhb = sh->ih[ib], xla = sh->il[ia], xlb = sh->il[ib];
  const float4 yha = sh->jh[ja], yhb = sh->jh[jb], yla = sh->jl[ja], ylb = sh->jl[jb];
  DF2 dx = df_sub(df2(yha.x, yla.x, yhb.x, ylb.x), df2(xha.x, xla.x, xhb.x, xlb.x));
  DF2 dy = df_sub(df2(yha.y, yla.y, yhb.y, ylb.y), df2(xha.y, xla.y, xhb.y, xlb.y));
  DF2 dz = df_sub(df2(yha.z, yla.z, yhb.z, ylb.z), df2(xha.z, xla.z, xhb.z, xlb.z));
  if (box.mi) {
    // (the image count times the box is exact in all its parts; what the sums of low parts
    // round off is kept for last: the same box for every pair, it would not average out)
    auto wrap = [](DF2 d, DF L, float iL, float t) {
      const float2 n = nb_images(d.h, iL);
      const DF2 s = df_two_sum(d.h, __fmul2_rn(n, f2(L.h))), u = df_two_sum(s.l, __fmul2_rn(n, f2(L.l)));
      const DF2 w = df_two_sum(u.h, d.l);
      d = df_fast_two_sum(s.h, w.h);
      d.l = __fadd2_rn(d.l, __ffma2_rn(n, f2(t), __fadd2_rn(u.l, w.l)));
      return d;
    };
    dx = wrap(dx, box.x, box.ix, box.tx);
    dy = wrap(dy, box.y, box.iy, box.ty);
    dz = wrap(dz, box.z, box.iz, box.tz);
  } else {
    dx = df_norm(dx);
    dy = df_norm(dy);
    dz = df_norm(dz);
  }
  const DF2 r2 = df_norm2(dx, dy, dz);
  const DF2 ir = df_rsqrt(r2);
  const DF2 r = df_norm(df_mul(r2, ir));
  const bool scaled = (ca | cb) & 2048u;   // (1-4 pairs: masked tiles only)
  const DF2 zero = df2(DF{0.f, 0.f}), one = df2(DF{1.f, 0.f});
  // LJ: energy and r dE/dr before switching
  DF2 Ev = zero, gv = zero;
  if (e.dovdw) {
    const float4 pa = sh->ip[ia], pb = sh->ip[ib], qa = sh->jp[ja], qb = sh->jp[jb];
    const DF2 R = df_norm(df_add(df2(pa.x, pa.z, pb.x, pb.z), df2(qa.x, qa.z, qb.x, qb.z)));
    const DF2 t = df_mul(R, ir), t2 = df_norm(df_sqr(t));
    const DF2 B = df_norm(df_mul(df_sqr(t2), t2)), A = df_sqr(B);
    DF2 eps = df_mul(df2(pa.y, pa.w, pb.y, pb.w), df2(qa.y, qa.w, qb.y, qb.w));
    if (scaled) eps = df_norm(df_mul(eps, df_select(ca & 2048u, cb & 2048u, df2(e.vdw14), one)));
    const DF2 AB = df_sub(A, B);
    Ev = df_norm(df_mul(eps, df_sub(AB, B)));
    gv = df_norm(df_mul(df_scale(eps, -12.f), df_norm(AB)));
    if (!SW) {
      const DF2 w = nb_beyond(r, e.vdwinner, e.vdwinner_t);
      if (w.h.x > 0.f || w.h.y > 0.f) {
        DF2 Sv, dS;
        nb_switch_df(r, w, e.vdwinvw2, Sv, dS);
        gv = df_add(df_mul(Sv, gv), df_mul(Ev, dS));
        Ev = df_mul(Ev, Sv);
      }
      const float ua = (r.h.x - e.vdwcut.h) + (r.l.x - e.vdwcut.l), ub = (r.h.y - e.vdwcut.h) + (r.l.y - e.vdwcut.l);
      bool va = ua < 0.f, vb = ub < 0.f;
      if (e.vdw_hard) {   // at an unswitched end of LJ: decided in FP64
        if (fabsf(ua) <= 2e-6f * e.vdwcut.h) va = sqrt(nb_r2_fp64(v, S, ibase + ia, sh->js[ja])) < k.vdwcut_d;
        if (fabsf(ub) <= 2e-6f * e.vdwcut.h) vb = sqrt(nb_r2_fp64(v, S, ibase + ib, sh->js[jb])) < k.vdwcut_d;
      }
      gv = df_select(va, vb, gv, zero);
      Ev = df_select(va, vb, Ev, zero);
    }
  }
  // Coulomb: energy and minus r dE/dr
  DF2 Ee = zero, fe = zero;
  if (ELEC != 0) {
    DF2 qq = df_mul(df2(xha.w, xla.w, xhb.w, xlb.w), df2(yha.w, yla.w, yhb.w, ylb.w));   // (i's charge carries the Coulomb constant)
    if (scaled) qq = df_mul(qq, df_select(ca & 2048u, cb & 2048u, df2(e.elec14), one));
    Ee = fe = df_norm(df_mul(qq, ir));
    if (ELEC == 3) {
      const DF2 w = nb_beyond(r, e.inner, e.inner_t);
      if (w.h.x > 0.f || w.h.y > 0.f) {
        DF2 Se, dS;
        nb_switch_df(r, w, e.invw2, Se, dS);
        if (SW) {   // one switch for both terms
          gv = df_add(df_mul(Se, gv), df_mul(Ev, dS));
          Ev = df_mul(Ev, Se);
        }
        fe = df_sub(df_mul(Se, Ee), df_mul(Ee, dS));
        Ee = df_mul(Ee, Se);
      }
    } else if (ELEC == 4) {
      // Steinbach & Brooks force switch, nonbonded.cpp:798-819
      const bool oa = r.h.x > e.inner.h, ob = r.h.y > e.inner.h;
      DF2 h = df_norm(df_sub(ir, df2(e.eshift)));
      h.l = __fadd2_rn(h.l, f2(-e.eshift_t));
      if (oa || ob) {
        DF2 c2 = df_norm(df_sub(df2(e.cut2), r2)), c3 = df_norm(df_add(df2(e.fsw_k), df_scale2(r2, 2.f)));
        c2.l = __fadd2_rn(c2.l, f2(e.cut2_t));
        c3.l = __fadd2_rn(c3.l, f2(e.fsw_t));
        // qq sA / r (C^2 - r^2)^2 (C^2 - 3 I^2 + 2 r^2)
        const DF2 f = df_mul(df_sqr(c2), c3);
        fe = df_select(oa, ob, df_mul(df_norm(df_mul(df2(e.sA), f)), fe), fe);
        // qq sA (C - r)^3 Q(r) / r
        DF2 c = df_norm(df_sub(df2(e.cut), r));
        c.l = __fadd2_rn(c.l, f2(e.cut_t));
        DF2 g = df_norm(df_add(df2(e.q2), df_mul(df2(e.q3), r)));
        g = df_norm(df_add(df2(e.q1), df_mul(g, r)));
        g = df_norm(df_add(df2(e.q0), df_mul(g, r)));
        g = df_mul(df_norm(df_mul(g, ir)), df_norm(df_mul(df_sqr(c), c)));
        h = df_select(oa, ob, df_mul(df2(e.sA), df_norm(g)), h);
      }
      Ee = df_mul(qq, df_norm(h));
    }
  }
  DF2 vir = df_sub(gv, fe);
  const float2 f = __fmul2_rn(vir.h, ir.h);
  sum.f = __fadd2_rn(sum.f, make_float2(fabsf(f.x), two ? fabsf(f.y) : 0.f));
  const bool la = fmaxf(fabsf(vir.h.x), fmaxf(fabsf(Ev.h.x), fabsf(Ee.h.x))) > kNbLarge;
  const bool lb = two && fmaxf(fabsf(vir.h.y), fmaxf(fabsf(Ev.h.y), fabsf(Ee.h.y))) > kNbLarge;
  if (la) nb_energy_large<ELEC>(v, k, S, ibase + ia, sh->js[ja], ca & 2048u);
  if (lb) nb_energy_large<ELEC>(v, k, S, ibase + ib, sh->js[jb], cb & 2048u);
  const bool ka = !la, kb = two && !lb;
  Ev = df_select(ka, kb, Ev, zero);
  Ee = df_select(ka, kb, Ee, zero);
  vir = df_select(ka, kb, vir, zero);
  df_acc(sum.vdw, Ev);
  df_acc(sum.elec, Ee);
  df_acc(sum.vir, vir);
}

// both halves' sum
__device__ __forceinline__ DF df_fold(DF2 x) { return df_add(DF{x.h.x, x.l.x}, DF{x.h.y, x.l.y}); }

// one block's atom of this lane into the shared rows (O: frame offset, with its rest)
__device__ __forceinline__ void nb_stage(float4* h, float4* l, float4* p, int row, const DevView& v, int slot,
                                         const DF* O, const float* rest, const DF* qscale) {
  const float4 x = v.xq[slot], rl = v.rlo[slot], par = v.par[slot];
  const float2 pl = v.plo[slot];
  DF X = DF{x.x, rl.x}, Y = DF{x.y, rl.y}, Z = DF{x.z, rl.z}, Q = DF{x.w, rl.w};
  if (O) {
    X.l += rest[0];
    Y.l += rest[1];
    Z.l += rest[2];
    X = df_norm(df_add(X, O[0]));
    Y = df_norm(df_add(Y, O[1]));
    Z = df_norm(df_add(Z, O[2]));
  }
  if (qscale) Q = df_norm(df_mul(Q, *qscale));
  h[row] = make_float4(X.h, Y.h, Z.h, Q.h);
  l[row] = make_float4(X.l, Y.l, Z.l, Q.l);
  p[row] = make_float4(par.x, par.y, pl.x, pl.y);
}

// per-tile FP32 sums enter 64-bit fixed point before they are combined, so a
// slot's total does not depend on how its tiles were grouped into work items
struct NBFix {
  long long fx, fy, fz;
};

__device__ __forceinline__ void nb_fix_in(const DevView& v, NBFix& F, const NBAcc& a) {
  fix_range(v.status, fabsf(a.fx) + fabsf(a.fy) + fabsf(a.fz));
  F.fx += fx32(a.fx);
  F.fy += fx32(a.fy);
  F.fz += fx32(a.fz);
}

__device__ __forceinline__ void nb_flush_fix(const DevView& v, int s, const NBFix& F) {
  atomic_add_ll(&v.facc[force_at(s, 0)], F.fx);
  atomic_add_ll(&v.facc[force_at(s, 1)], F.fy);
  atomic_add_ll(&v.facc[force_at(s, 2)], F.fz);
}

__device__ __forceinline__ void nb_flush(const DevView& v, int s, const NBAcc& a) {
  NBFix F = {0, 0, 0};
  nb_fix_in(v, F, a);
  nb_flush_fix(v, s, F);
}

// Whether the pass walks the j-atom groups: they fit their arrays, and they
// replace at least half of the tiles.  In a box of about twice the list radius
// nearly every tile needs a per-pair image and stays a tile (667 waters at 12 A:
// 45 of 2,016 tiles become 8 groups, same time either way); then the tile path
// serves all.
__device__ __forceinline__ bool nb_grouped(const DevView& v) { return v.cull_n[2] && 2 * v.cull_n[0] <= *v.ntiles; }

// Forces where the law does not end smoothly (a hard cutoff).  One warp per work
// item, grid-stride: the tiles left on the tile path, then the j-atom groups (cull:
// the last list build wrote them and they fit).
constexpr int kNbThreads = 256;
template <int ELEC>
__global__ void __launch_bounds__(kNbThreads, 4)
    k_nb_tiles(const __grid_constant__ DevView v, const __grid_constant__ NBConst k, int cull) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const bool grouped = cull && nb_grouped(v);
  const int nrest = grouped ? v.cull_n[0] : *v.ntiles;
  const int nitem = nrest + (grouped ? v.cull_n[1] : 0);
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nitem; w += nwarps) {
    NBAcc I = {0.f, 0.f, 0.f}, J = {0.f, 0.f, 0.f};
    int sjl;
    if (w < nrest) {
      const Tile T = v.tiles[grouped ? v.cull_rest[w] : w];
      sjl = T.bj * 32 + lane;
      const int si = T.bi * 32 + lane;
      const float4 xi = v.xq[si], pi = v.par[si], xj = j_in_i_frame(v, T, lane), pj = v.par[sjl];
      const float qi = xi.w * k.econv_diel;
      const SystemInfo& S = v.sys[v.slot_sys[T.bi]];
      const bool mi = T.flags & 1;
      if (tile_masked(T)) {
        unsigned ex, m14;
        tile_masks(v, T, lane, ex, m14);
        if (T.flags & 2) ex |= diag_exclusion(lane);
        nb_rot<ELEC, true, false>(v, k, S, lane, si, xi, pi, qi, ex, m14, xj, pj, mi, T.bj * 32, nullptr, I, J);
      } else {
        nb_rot<ELEC, false, false>(v, k, S, lane, si, xi, pi, qi, 0u, 0u, xj, pj, mi, T.bj * 32, nullptr, I, J);
      }
      nb_flush(v, si, I);
    } else {
      const int g = w - nrest, bi = v.cull_bi[g], si = bi * 32 + lane;
      const float4* gent = v.cull_ent + (size_t)g * 32;
      const float4 en = gent[lane];
      sjl = __float_as_int(en.w);
      const float4 xi = v.xq[si], pi = v.par[si];
      const float qi = xi.w * k.econv_diel;
      const SystemInfo& S = v.sys[v.slot_sys[bi]];
      float4 xj = make_float4(1.0e15f, 1.0e15f, 1.0e15f, 0.f), pj = make_float4(0.f, 0.f, 0.f, 0.f);
      if (sjl >= 0) {
        xj = v.xq[sjl];
        pj = v.par[sjl];
        xj.x += en.x;
        xj.y += en.y;
        xj.z += en.z;
      }
      nb_rot<ELEC, false, true>(v, k, S, lane, si, xi, pi, qi, 0u, 0u, xj, pj, false, 0, gent, I, J);
      nb_flush(v, si, I);
    }
    if (sjl >= 0) nb_flush(v, sjl, J);
  }
}

// appends this lane's pair to the warp's list where take (every lane calls this)
__device__ __forceinline__ void nb_list(unsigned short* list, int& np, bool take, unsigned code, unsigned lt) {
  const unsigned m = __ballot_sync(0xffffffffu, take);
  if (take) list[np + __popc(m & lt)] = (unsigned short)code;
  np += __popc(m);
}

// Energies: items as k_nb_force's, a CTA of two warps each (with one, 2,016 tiles of
// 667 waters left the chip with three warps a scheduler and a list of six rounds a warp).
// An item goes in four parts (a quarter of a tile's rotation; one 8-atom sub-block of the
// i block against two groups), two to a warp, so that the lists stay short.
constexpr int kNbEThreads = 64;
template <int ELEC, bool SW = false>
__global__ void __launch_bounds__(kNbEThreads, 8)
    k_nb_energy(const __grid_constant__ DevView v, const __grid_constant__ NBConst k, const __grid_constant__ NBEConst e,
                int cull) {
  pdl_sync();
  __shared__ NBEShared shared;
  NBEShared* sh = &shared;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  unsigned short* list = sh->pair[wp];
  const bool grouped = cull && nb_grouped(v);
  const int nrest = grouped ? v.cull_n[0] : *v.ntiles;
  const int nitem = nrest + (grouped ? v.cull_n[1] / 2 : 0);
  const float tol = 2e-6f * k.cut2, reach2 = k.cut2 * 1.00001f;
  for (int w = blockIdx.x; w < nitem; w += gridDim.x) {
    const bool tile = w < nrest;
    int bi;
    NBEBox box = {};
    unsigned ex = 0u, m14 = 0u;
    if (tile) {
      const Tile T = v.tiles[grouped ? v.cull_rest[w] : w];
      bi = T.bi;
      tile_masks(v, T, lane, ex, m14);
      if (T.flags & 2) ex |= diag_exclusion(lane);
      if (T.flags & 1) {
        const SystemInfo& S = v.sys[v.slot_sys[bi]];
        box = NBEBox{true, S.boxf[0], S.boxf[1], S.boxf[2], 1.f / S.boxf[0].h, 1.f / S.boxf[1].h, 1.f / S.boxf[2].h,
                     S.boxt[0], S.boxt[1], S.boxt[2]};
      }
      if (wp == 1) {
        const float o[3] = {T.ox, T.oy, T.oz};
        DF O[3];
        float t[3];
        df_offset(v, v.sys[v.slot_sys[bi]], bi, T.bj, o, O, t);
        nb_stage(sh->jh, sh->jl, sh->jp, lane, v, T.bj * 32 + lane, O, t, nullptr);
        sh->js[lane] = T.bj * 32 + lane;
      }
    } else {
      const int g = 2 * (w - nrest) + wp, row = threadIdx.x;
      bi = v.cull_bi[g];
      const float4 en = v.cull_ent[(size_t)g * 32 + lane];
      const int sj = __float_as_int(en.w);
      sh->js[row] = sj;
      if (sj >= 0) {
        const float o[3] = {en.x, en.y, en.z};
        DF O[3];
        float t[3];
        df_offset(v, v.sys[v.slot_sys[bi]], bi, sj >> 5, o, O, t);
        nb_stage(sh->jh, sh->jl, sh->jp, row, v, sj, O, t, nullptr);
      } else {
        sh->jh[row] = make_float4(1.0e15f, 1.0e15f, 1.0e15f, 0.f);   // (empty lanes: far away)
      }
    }
    const SystemInfo& S = v.sys[v.slot_sys[bi]];
    if (wp == 0) nb_stage(sh->ih, sh->il, sh->ip, lane, v, bi * 32 + lane, nullptr, nullptr, &e.econv);
    __syncthreads();
    // a tile's i atom of this lane; minus its two j atoms of a group pair
    const float4 xi = sh->ih[lane], ja = sh->jh[lane], jb = sh->jh[tile ? lane : 32 + lane];
    const float2 nx = make_float2(-ja.x, -jb.x), ny = make_float2(-ja.y, -jb.y), nz = make_float2(-ja.z, -jb.z);
    const DF2 zero = df2(DF{0.f, 0.f});
    NBESum sum = {zero, zero, zero, f2(0.f)};
    int np = 0;
#pragma unroll 1
    for (int s = 2 * wp; s < 2 * wp + 2; s++) {
      if (tile) {
#pragma unroll 4
        for (int kk = 8 * s; kk < 8 * s + 8; kk++) {
          const int row = (lane + kk) & 31;
          const float4 x = sh->jh[row];
          float dx = x.x - xi.x, dy = x.y - xi.y, dz = x.z - xi.z;
          if (box.mi) {
            constexpr float kRint = 12582912.f;
            dx = fmaf(fmaf(dx, -box.ix, kRint) - kRint, box.x.h, dx);
            dy = fmaf(fmaf(dy, -box.iy, kRint) - kRint, box.y.h, dy);
            dz = fmaf(fmaf(dz, -box.iz, kRint) - kRint, box.z.h, dz);
          }
          const float r2 = dx * dx + dy * dy + dz * dz;
          bool in = r2 <= k.cut2;
          const bool listed = !((ex >> kk) & 1u);
          // at the cutoff: decided in FP64
          if (listed && fabsf(r2 - k.cut2) <= tol) in = nb_r2_fp64(v, S, bi * 32 + lane, sh->js[row]) <= k.cut2_dd;
          nb_list(list, np, listed && in, lane | row << 5 | (((m14 >> kk) & 1u) << 11), lt);
        }
      } else {
        const float4 lo = v.sub[8 * bi + 2 * s], hi = v.sub[8 * bi + 2 * s + 1];
        float d2 = 3.0e38f;
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const float4 x = q ? jb : ja;
          const float gx = fmaxf(fmaxf(lo.x - x.x, x.x - hi.x), 0.f), gy = fmaxf(fmaxf(lo.y - x.y, x.y - hi.y), 0.f);
          const float gz = fmaxf(fmaxf(lo.z - x.z, x.z - hi.z), 0.f);
          d2 = fminf(d2, gx * gx + gy * gy + gz * gz);
        }
        if (__any_sync(0xffffffffu, d2 <= reach2)) {
#pragma unroll 4
          for (int kk = 0; kk < 8; kk++) {
            const int row = 8 * s + ((lane + kk) & 7);
            const float4 x = sh->ih[row];
            const float2 dx = __fadd2_rn(f2(x.x), nx), dy = __fadd2_rn(f2(x.y), ny), dz = __fadd2_rn(f2(x.z), nz);
            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            bool ina = r2.x <= k.cut2, inb = r2.y <= k.cut2;
            if (fminf(fabsf(r2.x - k.cut2), fabsf(r2.y - k.cut2)) <= tol) {
              if (fabsf(r2.x - k.cut2) <= tol) ina = nb_r2_fp64(v, S, bi * 32 + row, sh->js[lane]) <= k.cut2_dd;
              if (fabsf(r2.y - k.cut2) <= tol) inb = nb_r2_fp64(v, S, bi * 32 + row, sh->js[32 + lane]) <= k.cut2_dd;
            }
            nb_list(list, np, ina, row | lane << 5, lt);
            nb_list(list, np, inb, row | (32 + lane) << 5, lt);
          }
        }
      }
      // full rounds of two pairs a lane now, the rest with the next part
      const int n = s & 1 ? np : np & ~63;
      __syncwarp();
      for (int p = lane; p < n; p += 64) {
        const bool two = p + 32 < n;
        nb_energy_df2<ELEC, SW>(v, k, e, S, box, bi * 32, sh, list[p], list[two ? p + 32 : p], two, sum);
      }
      const unsigned short keep0 = list[min(n + lane, kNbList - 1)], keep1 = list[min(n + 32 + lane, kNbList - 1)];
      __syncwarp();
      np -= n;
      if (lane < np) list[lane] = keep0;
      if (lane + 32 < np) list[lane + 32] = keep1;
    }
    // (as the force passes check theirs: a call may come without forces)
    fix_range(v.status, sum.f.x + sum.f.y);
    // the lanes' sums meet in double-float and enter fixed point once per item
    const DF ev = df_warp_sum(df_fold(sum.vdw)), ee = df_warp_sum(df_fold(sum.elec)), vir = df_warp_sum(df_fold(sum.vir));
    const DF x = lane == 0 ? ev : (lane == 1 ? ee : vir);
    if (wp == 1 && lane < 3) sh->sum[lane] = x;
    __syncthreads();
    if (wp == 0 && lane < 3) {
      const DF y = df_add(x, sh->sum[lane]);
      long long* E = v.eacc + (size_t)v.slot_sys[bi] * E_NSLOTS;
      atomic_add_ll(&E[lane == 0 ? E_VDW : (lane == 1 ? E_ELEC : E_VIRIAL)], fix_energy_d((double)y.h + (double)y.l));
    }
  }
}

// ---------------------------------------------------------------------------
// Force-only pass (every dynamics step) where the law ends smoothly: LJ and
// Coulomb both go to zero at their cutoffs by a switch (NBConst::smooth), so a
// pair beyond them contributes exactly 0 by clamping the switch and no pair needs
// a decision at a cutoff.  Packed FP32x2 arithmetic throughout.
//  * Groups, two of a row at once (.x, .y): each lane holds a j atom of either,
//    the i block's atoms come from the warp's rows, 8 at a time (one sub-block of
//    the sorted order): a sub-block whose box at the current positions no held
//    atom reaches is skipped (on the solvated box half of the steps: a far j atom
//    reaches part of a 32-atom block only, and the list build puts j atoms that
//    reach the same sub-blocks together).  The i atoms' sums rotate within 8 lanes
//    and meet over the four 8-lane groups after each sub-block.
//  * Tiles (masked, diagonal, or with a per-pair image), step-packed: lane l
//    holds i atom l, the j atoms l + kk and l + kk + 1 come as one pair.
// Bound by the FMA pipe (a packed instruction holds it two cycles) in the steps and
// by the gathers and atomics of the j atoms in an item's rest, about half each.
// Solvated box, 22,489 atoms at 12 A: 88 us (scalar rotation of 32 x 32 items) ->
// 49 (packed, skipping) -> 46 us (j atoms by class); 8 copies 607 -> 314 -> 275 us.
// ---------------------------------------------------------------------------
enum NBLaw { kLawSame = 0, kLawSplit = 1, kLawForce = 2, kLawVdw = 3 };

// dE/dr / r of two pairs; QQ = -econv q q, SS the radius sums, EE = eps.
// Switch S = s^2, s = 1 - u^2 / w^2 clamped at 0, u = r - inner clamped at 0 (that difference
// is exact; r and the inner radius over a width rounded in FP32 move the shell by 7e-7 of it).
template <int LAW>
__device__ __forceinline__ float2 nb_law2(const NBConst& k, float2 r2, float2 QQ, float2 SS, float2 EE) {
  const float2 M1 = f2(-1.f);
  const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 ir2 = __fmul2_rn(ir, ir), r = __fmul2_rn(r2, ir);
  const float2 t2 = __fmul2_rn(__fmul2_rn(SS, SS), ir2);
  const float2 b6 = __fmul2_rn(__fmul2_rn(t2, t2), t2);
  const float2 eb = __fmul2_rn(EE, b6), ea = __fmul2_rn(eb, b6);      // eps B, eps A
  const float2 t = __ffma2_rn(eb, M1, ea), ev = __ffma2_rn(eb, M1, t);   // eps (A - B), eps (A - 2B)
  float2 u = __fadd2_rn(r, f2(-k.vdwinner_f));
  u = make_float2(fmaxf(u.x, 0.f), fmaxf(u.y, 0.f));
  float2 s = __ffma2_rn(__fmul2_rn(u, u), f2(-k.vdwinvw2_f), f2(1.f));
  s = make_float2(fmaxf(s.x, 0.f), fmaxf(s.y, 0.f));
  const float2 Sv = __fmul2_rn(__fmul2_rn(s, s), ir2);                                 // S / r^2
  const float2 nv = __fmul2_rn(__fmul2_rn(u, s), __fmul2_rn(ir, f2(-4.f * k.vdwinvw2_f)));   // S' / r
  if (LAW == kLawVdw) return __ffma2_rn(__fmul2_rn(t, f2(-12.f)), Sv, __fmul2_rn(ev, nv));
  const float2 e1 = __fmul2_rn(QQ, ir);   // -E_coulomb
  if (LAW == kLawSame) return __ffma2_rn(__ffma2_rn(t, f2(-12.f), e1), Sv, __fmul2_rn(__ffma2_rn(e1, M1, ev), nv));
  const float2 gv = __ffma2_rn(__fmul2_rn(t, f2(-12.f)), Sv, __fmul2_rn(ev, nv));
  if (LAW == kLawSplit) {
    u = __fadd2_rn(r, f2(-k.inner_f));
    u = make_float2(fmaxf(u.x, 0.f), fmaxf(u.y, 0.f));
    s = __ffma2_rn(__fmul2_rn(u, u), f2(-k.invw2_f), f2(1.f));
    s = make_float2(fmaxf(s.x, 0.f), fmaxf(s.y, 0.f));
    const float2 Se = __fmul2_rn(__fmul2_rn(s, s), ir2);
    const float2 ne = __fmul2_rn(__fmul2_rn(u, s), __fmul2_rn(ir, f2(4.f * k.invw2_f)));
    return __ffma2_rn(e1, Se, __ffma2_rn(e1, ne, gv));
  }
  // Steinbach & Brooks force switch, nonbonded.cpp:798-819
  float2 c = __ffma2_rn(r2, M1, f2(k.cut2));
  c = make_float2(fmaxf(c.x, 0.f), fmaxf(c.y, 0.f));
  const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(c, c), __ffma2_rn(r2, f2(2.f), f2(k.fsw_k))), f2(k.sA_f));
  const float2 m = make_float2(r.x > k.inner_f ? f.x : 1.f, r.y > k.inner_f ? f.y : 1.f);
  return __ffma2_rn(__fmul2_rn(e1, ir2), m, gv);
}

struct NBRows {
  union {
    struct {
      float4 xy[64], zq[64], se[64];   // tiles: step pairs of the j block, twice over
    };
    struct {
      float4 x[64];                    // groups: (x, y, z, q) of the i block, each sub-block twice over
      float2 p[64];                    // (LJ radius, sqrt(eps))
      float4 c[4], h[4];               // the sub-blocks' boxes: centres, half-extents
    };
  };
};

template <int LAW, bool MASKED, bool MI>
__device__ __forceinline__ void nb_tile2(const DevView& v, const NBConst& k, const Tile& T, int lane, NBRows& rs) {
  const int si = T.bi * 32 + lane, sj = T.bj * 32 + lane, l1 = (lane + 1) & 31;
  const float4 xi = v.xq[si], pi = v.par[si];
  const SystemInfo& S = v.sys[v.slot_sys[T.bi]];
  unsigned ex = 0u, m14 = 0u;
  if (MASKED) {
    tile_masks(v, T, lane, ex, m14);
    if (T.flags & 2) ex |= diag_exclusion(lane);
  }
  {
    const float4 x0 = j_in_i_frame(v, T, lane), p0 = v.par[sj];
    const float e0 = p0.y;
    const float x1 = __shfl_sync(0xffffffffu, x0.x, l1), y1 = __shfl_sync(0xffffffffu, x0.y, l1);
    const float z1 = __shfl_sync(0xffffffffu, x0.z, l1), q1 = __shfl_sync(0xffffffffu, x0.w, l1);
    const float s1 = __shfl_sync(0xffffffffu, p0.x, l1), e1 = __shfl_sync(0xffffffffu, e0, l1);
    __syncwarp();
    rs.xy[lane] = rs.xy[lane + 32] = make_float4(x0.x, x1, x0.y, y1);
    rs.zq[lane] = rs.zq[lane + 32] = make_float4(x0.z, z1, x0.w, q1);
    rs.se[lane] = rs.se[lane + 32] = make_float4(p0.x, s1, e0, e1);
    __syncwarp();
  }
  const float2 X = f2(-xi.x), Y = f2(-xi.y), Z = f2(-xi.z), Q = f2(-k.econv_diel * xi.w), R = f2(pi.x);
  const float2 E = f2(pi.y);
  float Lx = 0.f, Ly = 0.f, Lz = 0.f, iLx = 0.f, iLy = 0.f, iLz = 0.f;
  if (MI) {
    Lx = S.boxf[0].h; Ly = S.boxf[1].h; Lz = S.boxf[2].h;
    iLx = 1.f / Lx; iLy = 1.f / Ly; iLz = 1.f / Lz;
  }
  constexpr float kRint = 12582912.f;   // 1.5 2^23: adding and taking it off rounds to an integer
  float2 FX = f2(0.f), FY = f2(0.f), FZ = f2(0.f), JX = f2(0.f), JY = f2(0.f), JZ = f2(0.f);   // J: minus the sums
  const float4 *xy = rs.xy + lane, *zq = rs.zq + lane, *se = rs.se + lane;
#pragma unroll 2
  for (int kk = 0; kk < 32; kk += 2) {
    const float4 P = xy[kk], ZQ = zq[kk], SE = se[kk];
    float2 dx = __fadd2_rn(make_float2(P.x, P.y), X), dy = __fadd2_rn(make_float2(P.z, P.w), Y);
    float2 dz = __fadd2_rn(make_float2(ZQ.x, ZQ.y), Z);
    if (MI) {
      const float2 nx = __fadd2_rn(__ffma2_rn(dx, f2(iLx), f2(kRint)), f2(-kRint));
      const float2 ny = __fadd2_rn(__ffma2_rn(dy, f2(iLy), f2(kRint)), f2(-kRint));
      const float2 nz = __fadd2_rn(__ffma2_rn(dz, f2(iLz), f2(kRint)), f2(-kRint));
      dx = __ffma2_rn(nx, f2(-Lx), dx);
      dy = __ffma2_rn(ny, f2(-Ly), dy);
      dz = __ffma2_rn(nz, f2(-Lz), dz);
    }
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    float2 QQ = __fmul2_rn(Q, make_float2(ZQ.z, ZQ.w)), EE = __fmul2_rn(E, make_float2(SE.z, SE.w));
    if (MASKED) {
      const bool ma = (m14 >> kk) & 1u, mb = (m14 >> kk) & 2u;
      QQ = __fmul2_rn(QQ, make_float2(ma ? k.elec14 : 1.f, mb ? k.elec14 : 1.f));
      EE = __fmul2_rn(EE, make_float2(ma ? k.vdw14 : 1.f, mb ? k.vdw14 : 1.f));
    }
    float2 g = nb_law2<LAW>(k, r2, QQ, __fadd2_rn(R, make_float2(SE.x, SE.y)), EE);
    if (MASKED) g = make_float2((ex >> kk) & 1u ? 0.f : g.x, (ex >> kk) & 2u ? 0.f : g.y);
    FX = __ffma2_rn(g, dx, FX); FY = __ffma2_rn(g, dy, FY); FZ = __ffma2_rn(g, dz, FZ);
    JX = __ffma2_rn(g, dx, JX); JY = __ffma2_rn(g, dy, JY); JZ = __ffma2_rn(g, dz, JZ);
    ROT2(JX); ROT2(JY); ROT2(JZ);
  }
  const int lm = (lane + 31) & 31;
  const float jx = JX.x + __shfl_sync(0xffffffffu, JX.y, lm), jy = JY.x + __shfl_sync(0xffffffffu, JY.y, lm);
  const float jz = JZ.x + __shfl_sync(0xffffffffu, JZ.y, lm);
  nb_flush(v, si, NBAcc{FX.x + FX.y, FY.x + FY.y, FZ.x + FZ.y});
  nb_flush(v, sj, NBAcc{-jx, -jy, -jz});
}

// one pair of groups of row bi (entries en[0..63])
template <int LAW>
__device__ __forceinline__ void nb_groups2(const DevView& v, const NBConst& k, int bi, const float4* en, int lane,
                                           NBRows& rs) {
  const int si = bi * 32 + lane, row = (lane >> 3) * 16 + (lane & 7);
  const float4 xi = v.xq[si], pi = v.par[si];
  // the lane's two j atoms in i's frame (empty lanes parked far away)
  const float4 ea = en[lane], eb = en[32 + lane];
  const int sa = __float_as_int(ea.w), sb = __float_as_int(eb.w);
  float4 xa = make_float4(1.0e15f, 1.0e15f, 1.0e15f, 0.f), xb = xa, pa = make_float4(0.f, 0.f, 0.f, 0.f), pb = pa;
  if (sa >= 0) {
    xa = v.xq[sa];
    pa = v.par[sa];
    xa.x += ea.x; xa.y += ea.y; xa.z += ea.z;
  }
  if (sb >= 0) {
    xb = v.xq[sb];
    pb = v.par[sb];
    xb.x += eb.x; xb.y += eb.y; xb.z += eb.z;
  }
  float4 blo = make_float4(0.f, 0.f, 0.f, 0.f), bhi = blo;
  if (lane < 4) {
    blo = v.sub[8 * bi + 2 * lane];
    bhi = v.sub[8 * bi + 2 * lane + 1];
  }
  __syncwarp();
  if (lane < 4) {
    rs.c[lane] = make_float4(0.5f * (blo.x + bhi.x), 0.5f * (blo.y + bhi.y), 0.5f * (blo.z + bhi.z), 0.f);
    rs.h[lane] = make_float4(0.5f * (bhi.x - blo.x), 0.5f * (bhi.y - blo.y), 0.5f * (bhi.z - blo.z), 0.f);
  }
  rs.x[row] = rs.x[row + 8] = make_float4(xi.x, xi.y, xi.z, k.econv_diel * xi.w);
  rs.p[row] = rs.p[row + 8] = make_float2(pi.x, pi.y);
  __syncwarp();
  const float2 nx = make_float2(-xa.x, -xb.x), ny = make_float2(-xa.y, -xb.y), nz = make_float2(-xa.z, -xb.z);
  const float2 QN = make_float2(-xa.w, -xb.w), RS = make_float2(pa.x, pb.x);
  const float2 EN = make_float2(pa.y, pb.y);
  float2 FX = f2(0.f), FY = f2(0.f), FZ = f2(0.f);   // force on the held atoms along d = x_i - x_j
  float ix = 0.f, iy = 0.f, iz = 0.f;                // minus the sums of i atom `lane`
  // the sub-blocks that a held atom reaches (a hair more than the cutoff)
  const float reach2 = k.cut2 * 1.00001f;
  unsigned todo = 0u;
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const float4 c = rs.c[s], h = rs.h[s];
    float2 gx = __fadd2_rn(nx, f2(c.x)), gy = __fadd2_rn(ny, f2(c.y)), gz = __fadd2_rn(nz, f2(c.z));
    gx = make_float2(fmaxf(fabsf(gx.x) - h.x, 0.f), fmaxf(fabsf(gx.y) - h.x, 0.f));
    gy = make_float2(fmaxf(fabsf(gy.x) - h.y, 0.f), fmaxf(fabsf(gy.y) - h.y, 0.f));
    gz = make_float2(fmaxf(fabsf(gz.x) - h.z, 0.f), fmaxf(fabsf(gz.y) - h.z, 0.f));
    const float2 d2 = __ffma2_rn(gz, gz, __ffma2_rn(gy, gy, __fmul2_rn(gx, gx)));
    todo |= __any_sync(0xffffffffu, fminf(d2.x, d2.y) <= reach2) ? 1u << s : 0u;
  }
  const int src = (lane & 24) | ((lane + 1) & 7);
#pragma unroll 1
  for (; todo; todo &= todo - 1u) {
    const int s = __ffs(todo) - 1;
    const float4* xr = rs.x + s * 16 + (lane & 7);
    const float2* pr = rs.p + s * 16 + (lane & 7);
    float rx = 0.f, ry = 0.f, rz = 0.f;
#pragma unroll 4
    for (int kk = 0; kk < 8; kk++) {
      const float4 x = xr[kk];
      const float2 p = pr[kk];
      const float2 dx = __fadd2_rn(f2(x.x), nx), dy = __fadd2_rn(f2(x.y), ny), dz = __fadd2_rn(f2(x.z), nz);
      const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
      const float2 g = nb_law2<LAW>(k, r2, __fmul2_rn(QN, f2(x.w)), __fadd2_rn(RS, f2(p.x)), __fmul2_rn(EN, f2(p.y)));
      FX = __ffma2_rn(g, dx, FX); FY = __ffma2_rn(g, dy, FY); FZ = __ffma2_rn(g, dz, FZ);
      rx = fmaf(g.x, dx.x, rx); rx = fmaf(g.y, dx.y, rx);
      ry = fmaf(g.x, dy.x, ry); ry = fmaf(g.y, dy.y, ry);
      rz = fmaf(g.x, dz.x, rz); rz = fmaf(g.y, dz.y, rz);
      rx = __shfl_sync(0xffffffffu, rx, src);
      ry = __shfl_sync(0xffffffffu, ry, src);
      rz = __shfl_sync(0xffffffffu, rz, src);
    }
    // lane holds the sum of sub-block atom lane & 7 over its 8-lane group's j atoms
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      rx += __shfl_xor_sync(0xffffffffu, rx, o);
      ry += __shfl_xor_sync(0xffffffffu, ry, o);
      rz += __shfl_xor_sync(0xffffffffu, rz, o);
    }
    if ((lane >> 3) == s) {
      ix = rx;
      iy = ry;
      iz = rz;
    }
  }
  nb_flush(v, si, NBAcc{-ix, -iy, -iz});
  if (sa >= 0) nb_flush(v, sa, NBAcc{FX.x, FY.x, FZ.x});
  if (sb >= 0) nb_flush(v, sb, NBAcc{FX.y, FY.y, FZ.y});
}

constexpr int kNbFThreads = 128;
template <int LAW>
__global__ void __launch_bounds__(kNbFThreads, 6)
    k_nb_force(const __grid_constant__ DevView v, const __grid_constant__ NBConst k, int cull) {
  pdl_sync();
  __shared__ NBRows rows[kNbFThreads / 32];
  NBRows& rs = rows[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const bool grouped = cull && nb_grouped(v);
  const int nrest = grouped ? v.cull_n[0] : *v.ntiles;
  const int nitem = nrest + (grouped ? v.cull_n[1] / 2 : 0);
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nitem; w += nwarps) {
    if (w < nrest) {
      const Tile T = v.tiles[grouped ? v.cull_rest[w] : w];
      const bool mi = T.flags & 1;
      if (tile_masked(T)) {
        if (mi) nb_tile2<LAW, true, true>(v, k, T, lane, rs);
        else nb_tile2<LAW, true, false>(v, k, T, lane, rs);
      } else {
        if (mi) nb_tile2<LAW, false, true>(v, k, T, lane, rs);
        else nb_tile2<LAW, false, false>(v, k, T, lane, rs);
      }
    } else {
      const int g = 2 * (w - nrest);
      nb_groups2<LAW>(v, k, v.cull_bi[g], v.cull_ent + (size_t)g * 32, lane, rs);
    }
  }
}

// CTAs of T threads for the passes whose items take unequal times: `times` the other
// tile kernels' warps, no more than items, so that CTAs that end early make room for
// the next (k_nb_force, 8 copies of the solvated box: 336 -> 314 us; one copy 51 -> 49)
// items: per CTA
static int uneven_grid(const Context& c, int g, int T, int items, int times) {
  const long long want = (c.tile_cap + c.cull_cap / 64 + items - 1) / items;
  return (int)std::min<long long>((long long)times * g * (kNbThreads / T), want > 0 ? want : 1);
}

static void launch_nb_force(Context& c, const NBConst& k, int g) {
  DevView v = c.view();
  const int cull = c.cull_built ? 1 : 0;
  constexpr int T = kNbFThreads;
  g = uneven_grid(c, g, T, T / 32, 4);
  if (k.elecmode == 0) launch_pdl(c.stream, g, T, 0, k_nb_force<kLawVdw>, v, k, cull);
  else if (k.elecmode == 4) launch_pdl(c.stream, g, T, 0, k_nb_force<kLawForce>, v, k, cull);
  else if (k.samesw) launch_pdl(c.stream, g, T, 0, k_nb_force<kLawSame>, v, k, cull);
  else launch_pdl(c.stream, g, T, 0, k_nb_force<kLawSplit>, v, k, cull);
}

static void launch_nb_tiles(Context& c, const NBConst& k, int g) {
  DevView v = c.view();
  const int cull = c.cull_built ? 1 : 0;
  switch (k.elecmode) {
    case 0: launch_pdl(c.stream, g, kNbThreads, 0, k_nb_tiles<0>, v, k, cull); break;
    case 1: launch_pdl(c.stream, g, kNbThreads, 0, k_nb_tiles<1>, v, k, cull); break;
    case 3: launch_pdl(c.stream, g, kNbThreads, 0, k_nb_tiles<3>, v, k, cull); break;
    default: launch_pdl(c.stream, g, kNbThreads, 0, k_nb_tiles<4>, v, k, cull); break;
  }
}

static void launch_nb_energy(Context& c, const NBConst& k, int g) {
  DevView v = c.view();
  const int cull = c.cull_built ? 1 : 0;
  const NBEConst e = make_nbe_const(k);
  constexpr int T = kNbEThreads;
  g = uneven_grid(c, g, T, 1, 8);
  switch (k.elecmode) {
    case 0: launch_pdl(c.stream, g, T, 0, k_nb_energy<0>, v, k, e, cull); break;
    case 1: launch_pdl(c.stream, g, T, 0, k_nb_energy<1>, v, k, e, cull); break;
    case 3:
      if (k.samesw) launch_pdl(c.stream, g, T, 0, k_nb_energy<3, true>, v, k, e, cull);
      else launch_pdl(c.stream, g, T, 0, k_nb_energy<3>, v, k, e, cull);
      break;
    default: launch_pdl(c.stream, g, T, 0, k_nb_energy<4>, v, k, e, cull); break;
  }
}

int launch_df_records(Context& c) {
  c.kernel_launches += 1;
  const Spread sp = spread(c.nslots);
  launch_pdl(c.stream, sp.grid, sp.threads, 0, k_df_records, c.view(), c.d_charge.p, c.d_rlo.p, c.d_plo.p);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

// (the energies read the records of launch_df_records)
int launch_nb(Context& c, const NBConst& k, bool energy, bool forces) {
  const int g = tile_grid(c);
  if (forces) {
    c.kernel_launches += 1;
    if (k.smooth) launch_nb_force(c, k, g);
    else launch_nb_tiles(c, k, g);
  }
  if (energy) {
    c.kernel_launches += 1;
    launch_nb_energy(c, k, g);
  }
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

// fixed-point sorted accumulators -> N in original order; also flags overflow
__global__ void k_finalize_forces(DevView v, double* out, size_t stride, int add, double scale) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= v.nslots) return;
  int a = v.sorted_atom[s];
  if (a < 0) return;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    long long q = v.facc[force_at(s, c)];
    if (q >= (1ll << 62) || q <= -(1ll << 62)) atomicOr(v.status, (unsigned)ST_FIXED_OVERFLOW);
    double f = (double)q * (1.0 / kForceScale) * scale;
    if (add) out[a * stride + c] += f;
    else out[a * stride + c] = f;
  }
}

int launch_finalize_forces(Context& c, double* out, size_t stride_doubles, bool add, double scale) {
  c.kernel_launches += 1;
  DevView v = c.view();
  const Spread sp = spread(c.nslots);
  k_finalize_forces<<<sp.grid, sp.threads, 0, c.stream>>>(v, out, stride_doubles, add ? 1 : 0, scale);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

}  // namespace pdgpu
