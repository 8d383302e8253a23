// pdgpu_df.cuh — double-float arithmetic: a value as the unevaluated sum of two
// FP32 numbers, h + l with |l| a rounding of h (T. J. Dekker, "A floating-point
// technique for extending the available precision", Numer. Math. 18, 1971;
// D. E. Knuth, TAOCP vol. 2, 4.2.2: TwoSum).  About 45 significant bits on the
// FP32 pipe, which on this GPU has ~60 times the FP64 pipe's rate.  The _rn
// intrinsics keep the compiler from contracting or reordering the steps.
#pragma once

namespace pdgpu {

struct DF {
  float h, l;
};

// (host) the double x as a double-float
inline DF df_split(double x) {
  const float h = (float)x;
  return DF{h, (float)(x - (double)h)};
}

// what df_split leaves of x (a constant of all pairs of an energy: its error would not
// average out)
inline float df_rest(double x) {
  const DF s = df_split(x);
  return (float)(x - (double)s.h - (double)s.l);
}

__device__ __forceinline__ DF df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return DF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}

// |a| >= |b| (or a = 0)
__device__ __forceinline__ DF df_fast_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}

// The sums and products leave l unnormalised (it stays a few roundings of h);
// df_norm restores |l| <= ulp(h) / 2 where a chain of them needs it.
__device__ __forceinline__ DF df_norm(DF x) { return df_fast_two_sum(x.h, x.l); }
__device__ __forceinline__ DF df_neg(DF x) { return DF{-x.h, -x.l}; }
__device__ __forceinline__ DF df_add(DF x, DF y) {
  const DF s = df_two_sum(x.h, y.h);
  return DF{s.h, __fadd_rn(s.l, __fadd_rn(x.l, y.l))};
}
__device__ __forceinline__ DF df_sub(DF x, DF y) { return df_add(x, df_neg(y)); }
__device__ __forceinline__ DF df_mul(DF x, DF y) {
  const float p = __fmul_rn(x.h, y.h);
  float e = __fmaf_rn(x.h, y.h, -p);
  e = __fmaf_rn(x.h, y.l, e);
  return DF{p, __fmaf_rn(x.l, y.h, e)};
}
__device__ __forceinline__ DF df_scale(DF x, float f) {  // times an FP32 number
  const float p = __fmul_rn(x.h, f);
  return DF{p, __fmaf_rn(x.l, f, __fmaf_rn(x.h, f, -p))};
}
__device__ __forceinline__ DF df_scale2(DF x, float f) { return DF{x.h * f, x.l * f}; }  // f a power of two

// acc += x (the rounding errors of the running sum collect in acc.l)
__device__ __forceinline__ void df_acc(DF& acc, DF x) {
  const DF s = df_two_sum(acc.h, x.h);
  acc.h = s.h;
  acc.l = __fadd_rn(acc.l, __fadd_rn(s.l, x.l));
}

// x^2 + y^2 + z^2
__device__ __forceinline__ DF df_norm2(DF x, DF y, DF z) {
  const float px = __fmul_rn(x.h, x.h), py = __fmul_rn(y.h, y.h), pz = __fmul_rn(z.h, z.h);
  // 2 h l + l^2 + the rounding of h^2 (l^2 counts: a displacement's l is a
  // rounding of the coordinates, not of their difference)
  const float ex = __fmaf_rn(__fmaf_rn(2.f, x.h, x.l), x.l, __fmaf_rn(x.h, x.h, -px));
  const float ey = __fmaf_rn(__fmaf_rn(2.f, y.h, y.l), y.l, __fmaf_rn(y.h, y.h, -py));
  const float ez = __fmaf_rn(__fmaf_rn(2.f, z.h, z.l), z.l, __fmaf_rn(z.h, z.h, -pz));
  const DF s = df_two_sum(px, py), t = df_two_sum(s.h, pz);
  const float e = __fadd_rn(__fadd_rn(__fadd_rn(ex, ey), ez), __fadd_rn(s.l, t.l));
  return df_fast_two_sum(t.h, e);
}

// 1 / sqrt(x): the FP32 approximation y corrected by y (res / 2 + 3 res^2 / 8),
// res = 1 - x y^2 formed exactly to double-float (the series of (1 - res)^-1/2)
__device__ __forceinline__ DF df_rsqrt(DF x) {
  const float y = rsqrtf(x.h);
  const float w = __fmul_rn(y, y), we = __fmaf_rn(y, y, -w);
  const float p = __fmul_rn(x.h, w);
  float res = __fsub_rn(__fsub_rn(1.f, p), __fmaf_rn(x.h, w, -p));
  res = __fmaf_rn(-x.h, we, res);
  res = __fmaf_rn(-x.l, w, res);
  return df_fast_two_sum(y, __fmul_rn(__fmul_rn(y, res), __fmaf_rn(0.375f, res, 0.5f)));
}

// lane sums of a warp by a fixed butterfly order
__device__ __forceinline__ DF df_warp_sum(DF x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const DF y = DF{__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o)};
    x = df_add(x, y);
  }
  return df_norm(x);
}

// Two double-floats side by side in FP32x2 registers: the same steps, half the
// instructions (a packed one holds the FMA pipe two cycles).  Differences are formed
// as FMAs by -1, exact but for their one rounding: a negated operand would split the
// packed instruction into two scalar ones.
struct DF2 {
  float2 h, l;
};
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ DF2 df2(DF a) { return DF2{make_float2(a.h, a.h), make_float2(a.l, a.l)}; }
__device__ __forceinline__ DF2 df2(float ah, float al, float bh, float bl) {
  return DF2{make_float2(ah, bh), make_float2(al, bl)};
}
__device__ __forceinline__ DF2 df_two_sum(float2 a, float2 b) {
  const float2 s = __fadd2_rn(a, b), bb = fsub2(s, a);
  return DF2{s, __fadd2_rn(fsub2(a, fsub2(s, bb)), fsub2(b, bb))};
}
__device__ __forceinline__ DF2 df_two_diff(float2 a, float2 b) {   // a - b
  const float2 s = fsub2(a, b), bb = fsub2(s, a);
  return DF2{s, fsub2(fsub2(a, fsub2(s, bb)), __fadd2_rn(b, bb))};
}
__device__ __forceinline__ DF2 df_fast_two_sum(float2 a, float2 b) {
  const float2 s = __fadd2_rn(a, b);
  return DF2{s, fsub2(b, fsub2(s, a))};
}
__device__ __forceinline__ DF2 df_norm(DF2 x) { return df_fast_two_sum(x.h, x.l); }
__device__ __forceinline__ DF2 df_add(DF2 x, DF2 y) {
  const DF2 s = df_two_sum(x.h, y.h);
  return DF2{s.h, __fadd2_rn(s.l, __fadd2_rn(x.l, y.l))};
}
__device__ __forceinline__ DF2 df_sub(DF2 x, DF2 y) {
  const DF2 s = df_two_diff(x.h, y.h);
  return DF2{s.h, __fadd2_rn(s.l, fsub2(x.l, y.l))};
}
// x y - p, the rounding of p = x y
__device__ __forceinline__ float2 prod_err2(float2 x, float2 y, float2 p) {
  return __ffma2_rn(x, y, __fmul2_rn(p, make_float2(-1.f, -1.f)));
}
__device__ __forceinline__ DF2 df_mul(DF2 x, DF2 y) {
  const float2 p = __fmul2_rn(x.h, y.h);
  return DF2{p, __ffma2_rn(x.l, y.h, __ffma2_rn(x.h, y.l, prod_err2(x.h, y.h, p)))};
}
__device__ __forceinline__ DF2 df_sqr(DF2 x) {
  const float2 p = __fmul2_rn(x.h, x.h);
  return DF2{p, __ffma2_rn(__fadd2_rn(x.h, x.h), x.l, prod_err2(x.h, x.h, p))};
}
__device__ __forceinline__ DF2 df_scale(DF2 x, float f) {
  const float2 g = make_float2(f, f), p = __fmul2_rn(x.h, g);
  return DF2{p, __ffma2_rn(x.l, g, prod_err2(x.h, g, p))};
}
__device__ __forceinline__ DF2 df_scale2(DF2 x, float f) {   // f a power of two
  const float2 g = make_float2(f, f);
  return DF2{__fmul2_rn(x.h, g), __fmul2_rn(x.l, g)};
}
__device__ __forceinline__ DF2 df_select(bool a, bool b, DF2 x, DF2 y) {
  return DF2{make_float2(a ? x.h.x : y.h.x, b ? x.h.y : y.h.y), make_float2(a ? x.l.x : y.l.x, b ? x.l.y : y.l.y)};
}
__device__ __forceinline__ void df_acc(DF2& acc, DF2 x) {
  const DF2 s = df_two_sum(acc.h, x.h);
  acc.h = s.h;
  acc.l = __fadd2_rn(acc.l, __fadd2_rn(s.l, x.l));
}
__device__ __forceinline__ DF2 df_norm2(DF2 x, DF2 y, DF2 z) {
  const float2 px = __fmul2_rn(x.h, x.h), py = __fmul2_rn(y.h, y.h), pz = __fmul2_rn(z.h, z.h), two = make_float2(2.f, 2.f);
  // the three squares' 2 h l + l^2 and roundings, one chain
  float2 e = __fadd2_rn(__fadd2_rn(prod_err2(x.h, x.h, px), prod_err2(y.h, y.h, py)), prod_err2(z.h, z.h, pz));
  e = __ffma2_rn(__ffma2_rn(two, x.h, x.l), x.l, e);
  e = __ffma2_rn(__ffma2_rn(two, y.h, y.l), y.l, e);
  e = __ffma2_rn(__ffma2_rn(two, z.h, z.l), z.l, e);
  const DF2 s = df_two_sum(px, py), t = df_two_sum(s.h, pz);
  return df_fast_two_sum(t.h, __fadd2_rn(e, __fadd2_rn(s.l, t.l)));
}
__device__ __forceinline__ DF2 df_rsqrt(DF2 x) {
  const float2 y = make_float2(rsqrtf(x.h.x), rsqrtf(x.h.y)), one = make_float2(1.f, 1.f);
  const float2 w = __fmul2_rn(y, y), we = prod_err2(y, y, w);
  const float2 p = __fmul2_rn(x.h, w);
  float2 res = fsub2(fsub2(one, p), prod_err2(x.h, w, p));
  const float2 c = __ffma2_rn(x.l, w, __fmul2_rn(x.h, we));
  res = fsub2(res, c);
  const float2 q = __ffma2_rn(make_float2(0.375f, 0.375f), res, make_float2(0.5f, 0.5f));
  return df_fast_two_sum(y, __fmul2_rn(__fmul2_rn(y, res), q));
}

}  // namespace pdgpu
