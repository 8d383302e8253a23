// pdgpu_tile.cuh — pieces shared by the tile kernels: lane rotation of the j
// block, diagonal-tile exclusion, FP64 distance rechecks, tile masks and the
// FF_NonBonded pair law.
#pragma once
#include "pdgpu_context.cuh"

namespace pdgpu {

__device__ __forceinline__ unsigned diag_exclusion(int lane) {
  return ~((lane == 0) ? 0xffffffffu : ((1u << (32 - lane)) - 1u)) | 1u;
}

#define ROT(x) x = __shfl_sync(0xffffffffu, x, (lane + 1) & 31)
// an FP32x2 pair of a step-packed body, two lanes down
#define ROT2(p) p.x = __shfl_sync(0xffffffffu, p.x, (lane + 2) & 31); p.y = __shfl_sync(0xffffffffu, p.y, (lane + 2) & 31)

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// FP64 squared distance of two sorted slots from the original positions
static __device__ __noinline__ double r2_slots_fp64(const DevView& v, int sa, int sb) {
  int a = v.sorted_atom[sa], b = v.sorted_atom[sb];
  if (a < 0 || b < 0) return 1e300;
  double dx = v.pos[3 * b] - v.pos[3 * a], dy = v.pos[3 * b + 1] - v.pos[3 * a + 1],
         dz = v.pos[3 * b + 2] - v.pos[3 * a + 2];
  return dx * dx + dy * dy + dz * dz;
}

// j block of a tile moved into the i block's frame (centre offset in FP64)
__device__ __forceinline__ float4 j_in_i_frame(const DevView& v, const Tile& T, int lane) {
  float4 xj = v.xq[T.bj * 32 + lane];
  xj.x += T.ox;
  xj.y += T.oy;
  xj.z += T.oz;
  return xj;
}

// Whether a tile takes the masked body (bonded pairs or the diagonal).  The
// choice must be the same for all 32 lanes: the tile bodies rotate the j block
// with full-warp shuffles, which need every lane on the same path.
__device__ __forceinline__ bool tile_masked(const Tile& T) { return T.mask >= 0 || (T.flags & 2); }

// Whether every pair of the tile lies inside all cutoffs and switch radii of
// the list's components, with the list's displacement margin (set at build).
__device__ __forceinline__ bool tile_full(const Tile& T) { return (T.flags & 4) != 0; }

__device__ __forceinline__ void tile_masks(const DevView& v, const Tile& T, int lane, unsigned& ex, unsigned& m14) {
  ex = 0u;
  m14 = 0u;
  if (T.mask >= 0) {
    uint2 m = v.masks[T.mask * 32 + lane];
    ex = m.x;
    m14 = m.y;
  }
}

// centre of block bj seen from block bi, as double-floats, in the image the
// FP32 offset o was taken in, and what these leave of it (zero in open space): every pair
// of the tile takes the same offset, so its rounding would not average out
__device__ __forceinline__ void df_offset(const DevView& v, const SystemInfo& S, int bi, int bj, const float o[3],
                                          DF O[3], float rest[3]) {
  const float4 ci = v.cenf[bi], cj = v.cenf[bj];
  const float a[3] = {ci.x, ci.y, ci.z}, b[3] = {cj.x, cj.y, cj.z};
#pragma unroll
  for (int c = 0; c < 3; c++) {
    O[c] = df_two_sum(b[c], -a[c]);
    rest[c] = 0.f;
    if (S.periodic) {   // (n = 0, 1 or -1: times the box exact)
      const float n = -rintf((O[c].h - o[c]) / S.boxf[c].h);
      const DF s = df_two_sum(O[c].h, n * S.boxf[c].h), u = df_two_sum(O[c].l, s.l), w = df_two_sum(u.h, n * S.boxf[c].l);
      O[c] = df_fast_two_sum(s.h, w.h);
      rest[c] = __fadd_rn(__fadd_rn(u.l, w.l), n * S.boxt[c]);
    }
  }
}

// Whether every pair of the tile lies inside every GB cutoff and switch radius at
// the current positions: by the list's flag, or (lists without the displacement
// check carry none) from the blocks' radii where the cutoffs are far away
// (GBConst::far_inner).  xj: in the i block's frame; every lane calls this.
__device__ __forceinline__ bool tile_full_now(const GBConst& k, const Tile& T, const float4& xi, const float4& xj) {
  if (tile_full(T)) return true;
  if (k.far_inner <= 0.f) return false;
  float a = xi.x * xi.x + xi.y * xi.y + xi.z * xi.z, b = xj.x * xj.x + xj.y * xj.y + xj.z * xj.z;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  return sqrtf(a) + sqrtf(b) + 1e-3f < k.far_inner;   // |x_i| + |x_j| bounds every distance
}

// the exp-approximation switch is discontinuous: pairs within FP32 rounding of
// the threshold are decided in FP64
static __device__ __noinline__ bool gb_on_fp64(const DevView& v, int si, int sj, double thresh) {
  int a = v.sorted_atom[si], b = v.sorted_atom[sj];
  if (a < 0 || b < 0) return false;
  return -0.25 * r2_slots_fp64(v, si, sj) / (v.born[a] * v.born[b]) > thresh;
}

// 1 / x by the special-function unit alone (rcp.approx.ftz, ~1 ulp): the pair
// terms' reciprocals of r^2 (no multiply by the numerator 1 as __fdividef has)
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// bond order of an atom pair as PD's list stores it; 7 when not bonded
__device__ __forceinline__ int pair_bondorder(const DevView& v, int a, int b) {
  int lo = a < b ? a : b, hi = a < b ? b : a;
  int d = hi - lo;
  if (d == 0) return 0;
  if (d <= kBandWidth) {
    unsigned long long bit = 1ull << (d - 1);
    if (v.band_excl[lo] & bit) return 2;  // 1-1/1-2/1-3: all treated alike (excluded)
    if (v.band_14[lo] & bit) return 3;
    return 7;
  }
  int best = 7;
  for (int k = v.far_start[lo]; k < v.far_start[lo + 1]; k++)
    if (v.far_idx[k] == hi && v.far_bo[k] < best) best = v.far_bo[k];
  return best;
}

// FF_NonBonded's pair law in FP64 (Monte Carlo updates, energies of overlapping pairs)
template <int ELEC>
__device__ __forceinline__ void nb_pair(const NBConst& k, double r2, double rsum, double eps, double qq, double& ev,
                                        double& ee, double& r_dEdr) {
  const double r = sqrt(r2), invr = 1.0 / r;
  double dv = 0.0, de = 0.0, Ev = 0.0, Ee = 0.0;
  if (k.dovdw && r < k.vdwcut_d) {
    const double t = rsum * invr, t2 = t * t, B = t2 * t2 * t2, A = B * B;
    Ev = eps * (A - 2.0 * B);
    dv = -12.0 * eps * invr * (A - B);
    if (r > k.vdwinner_d) {
      const double u = r - k.vdwinner_d, sw = 1.0 - u * u * k.vdwinvw2_d, S = sw * sw;
      dv = S * dv + Ev * (-4.0 * k.vdwinvw2_d * u * sw);
      Ev *= S;
    }
  }
  if (ELEC == 1) {
    Ee = qq * invr;
    de = -Ee * invr;
  } else if (ELEC == 3) {
    Ee = qq * invr;
    de = -Ee * invr;
    if (r > k.inner_d) {
      const double u = r - k.inner_d, sw = 1.0 - u * u * k.invw2_d, S = sw * sw;
      de = S * de + Ee * (-4.0 * k.invw2_d * u * sw);
      Ee *= S;
    }
  } else if (ELEC == 4) {
    // Steinbach & Brooks force switch, nonbonded.cpp:798-819
    if (r > k.inner_d) {
      const double c2mr2 = k.cut2_d - r2;
      de = -qq * k.sA * invr * invr * c2mr2 * c2mr2 * (k.cut2_d - 3.0 * k.inner2_d + 2.0 * r2);
      Ee = -qq * (k.sA * r * (k.sB * invr * invr + k.sC + k.sD * r2 + k.sE * r2 * r2) - k.fsw_cutV);
    } else {
      de = -qq * invr * invr;
      Ee = qq * (invr - k.eshift);
    }
  }
  ev += Ev;
  ee += Ee;
  r_dEdr = r * (dv + de);
}

// FP64 squared distance of two sorted slots from the original positions
// (minimum image in a periodic box): pairs whose FP32 distance lies within 2e-6
// of a hard cutoff, and overlapping pairs' energies.
__device__ __forceinline__ double r2_fp64(const DevView& v, const SystemInfo& S, int sa, int sb) {
  int a = v.sorted_atom[sa], b = v.sorted_atom[sb];
  if (a < 0 || b < 0) return 1e300;
  double r2 = 0;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    double d = v.pos[3 * b + c] - v.pos[3 * a + c];
    if (S.periodic) d -= S.box[c] * rint(d * S.ibox[c]);
    r2 += d * d;
  }
  return r2;
}

}  // namespace pdgpu
