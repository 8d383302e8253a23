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

// Force part of the pair law in FP32 (same law as nb_pair): dE/dr divided by r.
// SW (energy switch on both terms over the same radii, the common PD setting):
// one switch factor serves LJ and Coulomb, dE/dr / r = S^2 (gv + ge) +
// (Ev + Ee) S' / r with S' = -4 u S / w^2.
template <int ELEC, bool SW = false>
__device__ __forceinline__ float nb_force_f(const NBConst& k, float r2, float rsum, float eps, float qq) {
  const float invr = rsqrtf(r2), ir2 = invr * invr;
  const float r = r2 * invr;
  if (SW) {
    const float t2 = rsum * rsum * ir2;
    const float B = t2 * t2 * t2, A = B * B;
    const bool vin = r < k.vdwcut_f;
    const float ev = vin ? eps * (A - 2.f * B) : 0.f;
    const float gv = vin ? -12.f * eps * ir2 * (A - B) : 0.f;
    const float Ee = qq * invr;
    const float u = fmaxf(r - k.inner_f, 0.f);
    const float sw = 1.f - u * u * k.invw2_f;
    return sw * sw * (gv - Ee * ir2) + (ev + Ee) * (-4.f * k.invw2_f * u * sw) * invr;
  }
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

// (ENERGY) what one warp keeps in shared memory for the energies of its work
// item: both blocks' atoms as double-floats in the i block's frame and the list
// of the pairs inside the cutoff
struct NBEShared {
  float4 ih[32], il[32], ip[32];   // (x, y, z, q) high and low parts; (R, sqrt(eps)) high and low
  float4 jh[32], jl[32], jp[32];
  int js[32];                      // j slots
  unsigned short pair[1024];       // i lane | j row << 5 | 1-4 << 10
};

// 32 rotation steps of one work item: lane i holds an i atom, (xj, pj) the
// lane's j atom already in i's frame.  Tiles: j slot jb + lane, per-pair image
// when mi.  GROUP: the j atoms of a group (slots in gent[].w, -1 = empty lane,
// parked far away), never masked, one image.  ENERGY: the pairs inside the
// cutoff are listed in sh->pair; returns their number.
template <int ELEC, bool MASKED, bool ENERGY, bool GROUP, bool SW>
__device__ __forceinline__ int nb_rot(const DevView& v, const NBConst& k, const SystemInfo& S, int lane, int si,
                                      const float4& xi, const float4& pi, float qi, unsigned ex, unsigned m14,
                                      float4 xj, float4 pj, bool mi_tile, int jb, const float4* gent, NBAcc& I,
                                      NBAcc& J, NBEShared* sh) {
  const bool mi = !GROUP && mi_tile;
  float Lx = 1.f, Ly = 1.f, Lz = 1.f;
  if (!GROUP && S.periodic) {
    Lx = (float)S.box[0]; Ly = (float)S.box[1]; Lz = (float)S.box[2];
  }
  const float iLx = 1.f / Lx, iLy = 1.f / Ly, iLz = 1.f / Lz;
  int np = 0;
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
                   (!SW && fabsf(r2 - k.vdwcut2) <= 2e-6f * k.vdwcut2))) {
      // at a hard cutoff: decide, and take the distance, in FP64 (FP64 work only on this branch)
      const int sjr = GROUP ? __float_as_int(gent[(lane + kk) & 31].w) : jb + ((lane + kk) & 31);
      const double d2 = nb_r2_fp64(v, S, si, sjr);
      in = d2 <= k.cut2_dd;
      r2 = (float)d2;
    }
    const bool take = listed && in;
    if (ENERGY) {
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take)
        sh->pair[np + __popc(m & ((1u << lane) - 1u))] =
            (unsigned short)(lane | (((lane + kk) & 31) << 5) | (MASKED && ((m14 >> kk) & 1u) ? 1024 : 0));
      np += __popc(m);
    }
    if (take) {
      const bool is14 = MASKED && ((m14 >> kk) & 1u);
      const float eps = pi.y * pj.y * (is14 ? k.vdw14 : 1.f);
      const float qq = qi * xj.w * (is14 ? k.elec14 : 1.f);
      const float fs = nb_force_f<ELEC, SW>(k, r2, pi.x + pj.x, eps, qq);
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
  return np;
}

// ---------------------------------------------------------------------------
// Pair energies.  FP32 cannot hold them (water's electrostatics cancel ~5000
// fold, and so do the force-switch polynomials), and the FP64 pipe is narrow:
// they are formed in double-float arithmetic (pdgpu_df.cuh, ~45 bits) from
// positions and parameters held as double-floats.  The rotation lists the pairs
// inside the cutoff (about a fifth of those it visits); the list is then dealt
// over the lanes, so the ~300 instructions of a pair's energy run on full warps.
// FP64 pair energies on the rotation itself, bound by the FP64 pipe, had taken
// 5.85 ms on the solvated 22,489 atoms at 15 A (force switch), 0.331 ms on 667
// waters at 12 A; this takes 0.472 and 0.046 ms, bound by FP32 issue.  Against
// 64-bit sums the energies are as close as before (within 2e-8 kcal/mol, one
// fixed-point rounding per item instead of one per lane).
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
  DF vdw, elec, vir;
};

// energies of one listed pair into the sums (same law as nb_pair)
template <int ELEC, bool SW>
__device__ __forceinline__ void nb_energy_df(const DevView& v, const NBConst& k, const NBEConst& e,
                                             const SystemInfo& S, bool mi, int ibase, const NBEShared* sh,
                                             unsigned code, NBESum& sum) {
  const int il = code & 31, jl = (code >> 5) & 31;
  const bool is14 = code & 1024u;
  const float4 xh = sh->ih[il], xl = sh->il[il], xp = sh->ip[il];
  const float4 yh = sh->jh[jl], yl = sh->jl[jl], yp = sh->jp[jl];
  DF dx = df_sub(DF{yh.x, yl.x}, DF{xh.x, xl.x});
  DF dy = df_sub(DF{yh.y, yl.y}, DF{xh.y, xl.y});
  DF dz = df_sub(DF{yh.z, yl.z}, DF{xh.z, xl.z});
  if (mi) {
    dx = df_add(dx, df_scale(S.boxf[0], -rintf(dx.h / S.boxf[0].h)));
    dy = df_add(dy, df_scale(S.boxf[1], -rintf(dy.h / S.boxf[1].h)));
    dz = df_add(dz, df_scale(S.boxf[2], -rintf(dz.h / S.boxf[2].h)));
  }
  const DF r2 = df_norm2(dx, dy, dz);
  const DF ir = df_rsqrt(r2);
  const DF r = df_norm(df_mul(r2, ir));
  const DF one = DF{1.f, 0.f};
  // LJ: energy and r dE/dr before switching
  DF Ev = DF{0.f, 0.f}, gv = Ev;
  DF u = df_sub(r, e.vdwcut);
  bool vin = e.dovdw && u.h + u.l < 0.f;
  if (e.dovdw && e.vdw_hard && fabsf(u.h) <= 2e-6f * e.vdwcut.h)   // at an unswitched end of LJ: decide in FP64
    vin = sqrt(nb_r2_fp64(v, S, ibase + il, sh->js[jl])) < k.vdwcut_d;
  if (vin) {
    const DF R = df_norm(df_add(DF{xp.x, xp.z}, DF{yp.x, yp.z}));
    const DF t = df_norm(df_mul(R, ir)), t2 = df_norm(df_mul(t, t));
    const DF B = df_norm(df_mul(df_mul(t2, t2), t2)), A = df_mul(B, B);
    DF eps = df_norm(df_mul(DF{xp.y, xp.w}, DF{yp.y, yp.w}));
    if (is14) eps = df_norm(df_mul(eps, e.vdw14));
    Ev = df_norm(df_mul(eps, df_norm(df_sub(A, df_scale2(B, 2.f)))));
    gv = df_norm(df_scale(df_mul(eps, df_norm(df_sub(A, B))), -12.f));
    if (!SW) {
      DF w = df_sub(r, e.vdwinner);
      if (w.h > 0.f) {
        w = df_norm(w);
        const DF wi = df_norm(df_mul(w, e.vdwinvw2));
        const DF sw = df_norm(df_sub(one, df_mul(w, wi)));
        const DF Sv = df_norm(df_mul(sw, sw));
        const DF dS = df_norm(df_scale2(df_mul(df_mul(wi, sw), r), -4.f));   // r S'
        gv = df_add(df_mul(Sv, gv), df_mul(Ev, dS));
        Ev = df_mul(Ev, Sv);
      }
    }
  }
  // Coulomb
  DF Ee = DF{0.f, 0.f}, ge = Ee;
  if (ELEC != 0) {
    DF qq = df_norm(df_mul(DF{xh.w, xl.w}, DF{yh.w, yl.w}));   // (i's charge carries the Coulomb constant)
    if (is14) qq = df_norm(df_mul(qq, e.elec14));
    Ee = df_norm(df_mul(qq, ir));
    ge = df_neg(Ee);
    if (ELEC == 3) {
      DF w = df_sub(r, e.inner);
      if (w.h > 0.f) {
        w = df_norm(w);
        const DF wi = df_norm(df_mul(w, e.invw2));
        const DF sw = df_norm(df_sub(one, df_mul(w, wi)));
        const DF Se = df_norm(df_mul(sw, sw));
        const DF dS = df_norm(df_scale2(df_mul(df_mul(wi, sw), r), -4.f));
        if (SW) {   // one switch for both terms
          gv = df_add(df_mul(Se, gv), df_mul(Ev, dS));
          Ev = df_mul(Ev, Se);
        }
        ge = df_add(df_mul(Se, ge), df_mul(Ee, dS));
        Ee = df_mul(Ee, Se);
      }
    } else if (ELEC == 4) {
      // Steinbach & Brooks force switch, nonbonded.cpp:798-819
      if (df_sub(r, e.inner).h > 0.f) {
        const DF c2 = df_norm(df_sub(e.cut2, r2));
        // -qq sA / r (C^2 - r^2)^2 (C^2 - 3 I^2 + 2 r^2)
        const DF f = df_norm(df_mul(df_mul(c2, c2), df_norm(df_add(e.fsw_k, df_scale2(r2, 2.f)))));
        ge = df_neg(df_mul(df_norm(df_mul(e.sA, f)), Ee));
        // -qq (sA r (sB / r^2 + sC + sD r^2 + sE r^4) - V(C))
        DF h = df_norm(df_add(e.sD, df_mul(e.sE, r2)));
        h = df_norm(df_add(e.sC, df_mul(h, r2)));
        h = df_norm(df_add(df_mul(h, r), df_mul(e.sB, ir)));
        Ee = df_neg(df_mul(qq, df_norm(df_sub(df_mul(e.sA, h), e.cutV))));
      } else {
        Ee = df_mul(qq, df_norm(df_sub(ir, e.eshift)));
      }
    }
  }
  df_acc(sum.vdw, df_norm(Ev));
  df_acc(sum.elec, df_norm(Ee));
  df_acc(sum.vir, df_norm(df_add(gv, ge)));
}

// one block's atom of this lane into the shared rows (O: frame offset)
__device__ __forceinline__ void nb_stage(float4* h, float4* l, float4* p, int row, const DevView& v, int slot,
                                         const DF* O, const DF* qscale) {
  const float4 x = v.xq[slot], rl = v.rlo[slot], par = v.par[slot];
  const float2 pl = v.plo[slot];
  DF X = DF{x.x, rl.x}, Y = DF{x.y, rl.y}, Z = DF{x.z, rl.z}, Q = DF{x.w, rl.w};
  if (O) {
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

// One warp per work item, grid-stride: the tiles left on the tile path, then the
// j-atom groups (cull: the last list build wrote them and they fit).  The energy
// kernel's CTAs hold 4 warps (each warp keeps 5 KB of shared memory).
constexpr int kNbThreads = 256, kNbEThreads = 128;
template <int ELEC, bool ENERGY, bool SW = false>
__global__ void __launch_bounds__(ENERGY ? kNbEThreads : kNbThreads, ENERGY ? 5 : 4)
    k_nb_tiles(const __grid_constant__ DevView v, const __grid_constant__ NBConst k, const __grid_constant__ NBEConst e,
               int cull) {
  pdl_sync();
  __shared__ NBEShared shared[ENERGY ? kNbEThreads / 32 : 1];
  NBEShared* sh = ENERGY ? &shared[threadIdx.x >> 5] : nullptr;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const bool grouped = cull && nb_grouped(v);
  const int nrest = grouped ? v.cull_n[0] : *v.ntiles;
  const int nitem = nrest + (grouped ? v.cull_n[1] : 0);
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nitem; w += nwarps) {
    NBAcc I = {0.f, 0.f, 0.f}, J = {0.f, 0.f, 0.f};
    int bi, sjl, np;
    bool mi = false;
    float o[3];
    if (w < nrest) {
      const Tile T = v.tiles[grouped ? v.cull_rest[w] : w];
      bi = T.bi;
      sjl = T.bj * 32 + lane;
      const int si = T.bi * 32 + lane;
      const float4 xi = v.xq[si], pi = v.par[si];
      const float qi = xi.w * k.econv_diel;
      const SystemInfo& S = v.sys[v.slot_sys[T.bi]];
      unsigned ex = 0u, m14 = 0u;
      if (T.mask >= 0) {
        uint2 m = v.masks[T.mask * 32 + lane];
        ex = m.x;
        m14 = m.y;
      }
      if (T.flags & 2) ex |= diag_exclusion(lane);
      // j positions moved into i's frame (the tile's centre offset, periodic image included)
      float4 xj = v.xq[sjl];
      const float4 pj = v.par[sjl];
      o[0] = T.ox;
      o[1] = T.oy;
      o[2] = T.oz;
      xj.x += T.ox;
      xj.y += T.oy;
      xj.z += T.oz;
      mi = T.flags & 1;
      if (tile_masked(T))
        np = nb_rot<ELEC, true, ENERGY, false, SW>(v, k, S, lane, si, xi, pi, qi, ex, m14, xj, pj, mi, T.bj * 32,
                                                   nullptr, I, J, sh);
      else
        np = nb_rot<ELEC, false, ENERGY, false, SW>(v, k, S, lane, si, xi, pi, qi, ex, m14, xj, pj, mi, T.bj * 32,
                                                    nullptr, I, J, sh);
      nb_flush(v, si, I);
    } else {
      const int g = w - nrest;
      bi = v.cull_bi[g];
      const float4* gent = v.cull_ent + (size_t)g * 32;
      const float4 en = gent[lane];
      sjl = __float_as_int(en.w);
      o[0] = en.x;
      o[1] = en.y;
      o[2] = en.z;
      const int si = bi * 32 + lane;
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
      np = nb_rot<ELEC, false, ENERGY, true, SW>(v, k, S, lane, si, xi, pi, qi, 0u, 0u, xj, pj, false, 0, gent, I, J,
                                                 sh);
      nb_flush(v, si, I);
    }
    if (sjl >= 0) nb_flush(v, sjl, J);
    if (ENERGY) {
      const SystemInfo& S = v.sys[v.slot_sys[bi]];
      nb_stage(sh->ih, sh->il, sh->ip, lane, v, bi * 32 + lane, nullptr, &e.econv);
      sh->js[lane] = sjl;
      if (sjl >= 0) {
        DF O[3];
        df_offset(v, S, bi, sjl >> 5, o, O);
        nb_stage(sh->jh, sh->jl, sh->jp, lane, v, sjl, O, nullptr);
      }
      __syncwarp();
      NBESum sum = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      for (int p = lane; p < np; p += 32) nb_energy_df<ELEC, SW>(v, k, e, S, mi, bi * 32, sh, sh->pair[p], sum);
      // the lanes' sums meet in double-float and enter fixed point once per item
      const DF ev = df_warp_sum(sum.vdw), ee = df_warp_sum(sum.elec), vir = df_warp_sum(sum.vir);
      const DF x = lane == 0 ? ev : (lane == 1 ? ee : vir);
      if (lane < 3) {
        long long* E = v.eacc + (size_t)v.slot_sys[bi] * E_NSLOTS;
        atomic_add_ll(&E[lane == 0 ? E_VDW : (lane == 1 ? E_ELEC : E_VIRIAL)], fix_energy_d((double)x.h + (double)x.l));
      }
      __syncwarp();
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
// Switch S = s^2, s = 1 - u^2 clamped at 0, u = (r - inner) / w clamped at 0.
template <int LAW>
__device__ __forceinline__ float2 nb_law2(const NBConst& k, float2 r2, float2 QQ, float2 SS, float2 EE) {
  const float2 M1 = f2(-1.f);
  const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 ir2 = __fmul2_rn(ir, ir), r = __fmul2_rn(r2, ir);
  const float2 t2 = __fmul2_rn(__fmul2_rn(SS, SS), ir2);
  const float2 b6 = __fmul2_rn(__fmul2_rn(t2, t2), t2);
  const float2 eb = __fmul2_rn(EE, b6), ea = __fmul2_rn(eb, b6);      // eps B, eps A
  const float2 t = __ffma2_rn(eb, M1, ea), ev = __ffma2_rn(eb, M1, t);   // eps (A - B), eps (A - 2B)
  float2 u = __ffma2_rn(r, f2(k.vdwiw_f), f2(-k.vdwinner_iw_f));
  u = make_float2(fmaxf(u.x, 0.f), fmaxf(u.y, 0.f));
  float2 s = __ffma2_rn(__fmul2_rn(u, u), M1, f2(1.f));
  s = make_float2(fmaxf(s.x, 0.f), fmaxf(s.y, 0.f));
  const float2 Sv = __fmul2_rn(__fmul2_rn(s, s), ir2);                                 // S / r^2
  const float2 nv = __fmul2_rn(__fmul2_rn(u, s), __fmul2_rn(ir, f2(-4.f * k.vdwiw_f)));   // S' / r
  if (LAW == kLawVdw) return __ffma2_rn(__fmul2_rn(t, f2(-12.f)), Sv, __fmul2_rn(ev, nv));
  const float2 e1 = __fmul2_rn(QQ, ir);   // -E_coulomb
  if (LAW == kLawSame) return __ffma2_rn(__ffma2_rn(t, f2(-12.f), e1), Sv, __fmul2_rn(__ffma2_rn(e1, M1, ev), nv));
  const float2 gv = __ffma2_rn(__fmul2_rn(t, f2(-12.f)), Sv, __fmul2_rn(ev, nv));
  if (LAW == kLawSplit) {
    u = __ffma2_rn(r, f2(k.iw_f), f2(-k.inner_iw_f));
    u = make_float2(fmaxf(u.x, 0.f), fmaxf(u.y, 0.f));
    s = __ffma2_rn(__fmul2_rn(u, u), M1, f2(1.f));
    s = make_float2(fmaxf(s.x, 0.f), fmaxf(s.y, 0.f));
    const float2 Se = __fmul2_rn(__fmul2_rn(s, s), ir2);
    const float2 ne = __fmul2_rn(__fmul2_rn(u, s), __fmul2_rn(ir, f2(4.f * k.iw_f)));
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

static void launch_nb_force(Context& c, const NBConst& k, int g) {
  DevView v = c.view();
  const int cull = c.cull_built ? 1 : 0;
  constexpr int T = kNbFThreads;
  // four times the other tile kernels' warps (no more than items): the items
  // take unequal numbers of steps, and CTAs that end early make room for the next
  // (8 copies of the solvated box: 336 -> 314 us; one copy 51 -> 49)
  const long long want = (c.tile_cap + c.cull_cap / 64 + 3) / 4;
  g = (int)std::min<long long>(4LL * g * (256 / T), want > 0 ? want : 1);
  if (k.elecmode == 0) launch_pdl(c.stream, g, T, 0, k_nb_force<kLawVdw>, v, k, cull);
  else if (k.elecmode == 4) launch_pdl(c.stream, g, T, 0, k_nb_force<kLawForce>, v, k, cull);
  else if (k.samesw) launch_pdl(c.stream, g, T, 0, k_nb_force<kLawSame>, v, k, cull);
  else launch_pdl(c.stream, g, T, 0, k_nb_force<kLawSplit>, v, k, cull);
}

template <bool E>
static void launch_nb_mode(Context& c, const NBConst& k, int g) {
  DevView v = c.view();
  const int cull = c.cull_built ? 1 : 0;
  const NBEConst e = make_nbe_const(k);
  constexpr int T = E ? kNbEThreads : kNbThreads;
  g *= kNbThreads / T;
  switch (k.elecmode) {
    case 0: launch_pdl(c.stream, g, T, 0, k_nb_tiles<0, E>, v, k, e, cull); break;
    case 1: launch_pdl(c.stream, g, T, 0, k_nb_tiles<1, E>, v, k, e, cull); break;
    case 3:
      if (E && k.samesw) launch_pdl(c.stream, g, T, 0, k_nb_tiles<3, true, true>, v, k, e, cull);
      else launch_pdl(c.stream, g, T, 0, k_nb_tiles<3, E>, v, k, e, cull);
      break;
    default: launch_pdl(c.stream, g, T, 0, k_nb_tiles<4, E>, v, k, e, cull); break;
  }
}

int launch_df_records(Context& c) {
  const Spread sp = spread(c.nslots);
  launch_pdl(c.stream, sp.grid, sp.threads, 0, k_df_records, c.view(), c.d_charge.p, c.d_rlo.p, c.d_plo.p);
  return cudaGetLastError() == cudaSuccess ? PDGPU_OK : PDGPU_ERR_CUDA;
}

int launch_nb(Context& c, const NBConst& k, bool energy) {
  c.kernel_launches += 1;
  int g = tile_grid(c);
  if (energy) {
    c.kernel_launches += 1;
    launch_df_records(c);
    launch_nb_mode<true>(c, k, g);
  } else if (k.smooth) {
    launch_nb_force(c, k, g);
  } else {
    launch_nb_mode<false>(c, k, g);
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
