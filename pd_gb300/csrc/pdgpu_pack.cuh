// pdgpu_pack.cuh — one slot's packed record at the current positions.
#pragma once
#include "pdgpu_context.cuh"

namespace pdgpu {

// boxes of each 8 slots at the packed positions (a padding slot widens its box:
// it never hides an atom); every lane of the warp calls this
__device__ __forceinline__ void write_sub(const DevView& v, int s, const float4& o) {
  float4 lo = o, hi = o;
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, d));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, d));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, d));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, d));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, d));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, d));
  }
  if ((s & 7) == 0) {
    v.sub[s >> 2] = lo;
    v.sub[(s >> 2) + 1] = hi;
  }
}

// the block's radius about its centre (padding apart); every lane of the warp calls this
__device__ __forceinline__ void write_radius(const DevView& v, int s, int a, const float4& o) {
  float r2 = a >= 0 ? o.x * o.x + o.y * o.y + o.z * o.z : 0.f;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, d));
  if ((s & 31) == 0) v.brad[s >> 5] = sqrtf(r2) * 1.00001f;
}

// slot s of atom a (-1: padding) at FP64 position x -> FP32 offset from the block centre
__device__ __forceinline__ float4 packed_slot(const DevView& v, const SystemInfo& S, const double* charge, int s, int a,
                                              const double* x, const double c[3]) {
  // padding slot: zero parameters, parked far away from everything and each other
  if (a < 0) return make_float4(1.0e6f * (float)(1 + (s & 31)), 1.0e6f * (float)(1 + (s >> 5)), -1.0e6f, 0.f);
  double r[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double d = x[k] - c[k];
    if (S.periodic) d -= S.box[k] * rint(d * S.ibox[k]);
    r[k] = d;
  }
  return make_float4((float)r[0], (float)r[1], (float)r[2], (float)charge[a]);
}

// check2: squared skin limit (0 = no skin check); full2: squared limit that keeps
// tiles flagged full valid (0 = none flagged), checked where the skin check is not
// cull: the NB j-atom groups are in use (the displacement check always runs)
struct PackArgs {
  const double* charge;
  StepClear clear;
  float check2, full2;
  long long npairs_all;
  int cull;
  int gb;   // the GB passes need the blocks' radii
};
PackArgs pack_args(const Context& c, float check_disp);
inline float skin_disp(const Context& c) { return c.lp.check_skin ? (float)(0.5 * c.lp.Padding) : 0.f; }

// slot s of atom a (-1: padding) at position x; every lane of the warp calls this
__device__ __forceinline__ void pack_slot(const DevView& v, const PackArgs& P, int s, int a, const double* x) {
  const int b = s >> 5;
  const SystemInfo& S = v.sys[v.slot_sys[b]];
  const double c[3] = {v.center[3 * b], v.center[3 * b + 1], v.center[3 * b + 2]};
  const float4 o = packed_slot(v, S, P.charge, s, a, x, c);
  if (a >= 0) {
    // (in open space, when every block pair of every system is a tile, no pair
    // can leave the list; in a periodic box the tile images still depend on it)
    const bool skin = P.check2 > 0.f && (S.periodic || (long long)*v.ntiles < P.npairs_all || P.cull);
    const float lim = skin ? P.check2 : P.full2;
    if (lim > 0.f) {
      float4 q = v.rel0[s];
      float dx = o.x - q.x, dy = o.y - q.y, dz = o.z - q.z;
      if (dx * dx + dy * dy + dz * dz > lim) atomicOr(v.status, (unsigned)ST_STALE_LIST);
    }
  }
  v.xq[s] = o;
  if (P.cull) write_sub(v, s, o);
  if (P.gb) write_radius(v, s, a, o);
  step_clear(P.clear, v, s);
}

}  // namespace pdgpu
