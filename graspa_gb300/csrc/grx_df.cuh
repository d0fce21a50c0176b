// grx_df.cuh -- double-float ("float-float") arithmetic on the FP32 pipe.
//
// A value is an unevaluated sum hi + lo of two floats (about 48 significant bits).
// The error-free transformations are the classical ones: TwoSum (Knuth, TAOCP
// vol. 2, 4.2.2), FastTwoSum (Dekker 1971) and TwoProduct via fused multiply-add
// (the fma residual a*b - fl(a*b) is exact). Products and sums follow the
// double-double algorithms of Hida, Li and Bailey (QD library, 2001), restated
// here for float pairs. On GB300 one FP64 instruction issues at 1/64 of the FP32
// rate, so these 7-11 FP32 instructions per operation are several times cheaper
// than FP64 while keeping ~1e-14 relative accuracy.
#pragma once

#include <cstdint>

namespace grx {

struct df {
  float hi, lo;
};

// A float as a double by its bits (the conversion instruction issues at the FP64 rate).
__device__ __forceinline__ double wide(float x) {
  const unsigned b = __float_as_uint(x);
  if ((b & 0x7f800000u) - 0x00800000u >= 0x7f000000u) return (double)x;  // zero, below normal, inf, NaN
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

__device__ __forceinline__ double df_to(df a) { return wide(a.hi) + wide(a.lo); }

__device__ __forceinline__ df fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  const float e = __fsub_rn(b, __fsub_rn(s, a));
  return {s, e};
}

// A double as a float pair by its bits: the upper 24 significant bits rounded to nearest, the signed
// remainder of 29 bits as a float. The same pair as rounding and subtracting (ties aside), whose
// conversions and subtraction issue at the FP64 rate, 64 cycles a warp each.
__device__ __forceinline__ df df_from(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned e = (hi >> 20) & 0x7ffu;
  if (e - 960u >= 190u) {  // outside the range of two normal floats: zero, tiny, huge, inf, NaN
    const float h = __double2float_rn(x);
    return {h, __double2float_rn(x - (double)h)};
  }
  const unsigned sign = hi & 0x80000000u;
  const unsigned top = __funnelshift_l(lo, (hi & 0x7fffffffu) - (896u << 20), 3);
  const float h = __uint_as_float(sign | (top + ((lo >> 28) & 1u)));
  const float l = __fmul_rn((float)((int)(lo << 3) >> 3), __uint_as_float(sign | (e - 948u) << 23));
  return {h, l};
}

__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}

__device__ __forceinline__ df two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}

// a + b with the error bound relative to |a| + |b| (no cancellation guarantee)
__device__ __forceinline__ df df_add(df a, df b) {
  df s = two_sum(a.hi, b.hi);
  s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ df df_add_f(df a, float b) {
  df s = two_sum(a.hi, b);
  s.lo = __fadd_rn(s.lo, a.lo);
  return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ df df_mul(df a, df b) {
  df p = two_prod(a.hi, b.hi);
  p.lo = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo));
  return fast_two_sum(p.hi, p.lo);
}

__device__ __forceinline__ df df_mul_f(df a, float b) {
  df p = two_prod(a.hi, b);
  p.lo = __fmaf_rn(a.lo, b, p.lo);
  return fast_two_sum(p.hi, p.lo);
}

// a += h + l, a kept as an unnormalised pair: the exact error of the hi sum joins the low part.
__device__ __forceinline__ void df_accumulate(df& a, float h, float l) {
  const df s = two_sum(a.hi, h);
  a.hi = s.hi;
  a.lo = __fadd_rn(a.lo, __fadd_rn(s.lo, l));
}

// a += x y, a kept as an unnormalised pair: 12 instructions where df_mul and df_add take 20.
__device__ __forceinline__ void df_mac(df& a, df x, df y) {
  const df p = two_prod(x.hi, y.hi);
  df_accumulate(a, p.hi, __fmaf_rn(x.hi, y.lo, __fmaf_rn(x.lo, y.hi, p.lo)));
}

// x^2 + y^2 + z^2 for x = xh + xl etc., where xh carries few significant bits and
// |xl| is tiny: exact squares of the hi parts via TwoProduct, cross terms in FP32.
__device__ __forceinline__ df df_norm2_split(float3 h, float3 l) {
  df sx = two_prod(h.x, h.x), sy = two_prod(h.y, h.y), sz = two_prod(h.z, h.z);
  const float cross = __fmaf_rn(2.0f * h.x, l.x, __fmaf_rn(2.0f * h.y, l.y, __fmul_rn(2.0f * h.z, l.z)));
  const float small = __fmaf_rn(l.x, l.x, __fmaf_rn(l.y, l.y, __fmul_rn(l.z, l.z)));
  df s = two_sum(sx.hi, sy.hi);
  df t = two_sum(s.hi, sz.hi);
  const float lo = __fadd_rn(__fadd_rn(__fadd_rn(s.lo, t.lo), __fadd_rn(sx.lo, __fadd_rn(sy.lo, sz.lo))),
                             __fadd_rn(cross, small));
  return fast_two_sum(t.hi, lo);
}

// a < b for double-float values (b normalised)
__device__ __forceinline__ bool df_lt(df a, df b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }

// 1 / a to double-float accuracy (one Newton step on the FP32 reciprocal)
__device__ __forceinline__ df df_recip(df a) {
  const float r = __frcp_rn(a.hi);
  // e = 1 - a*r computed in double-float, then r + r*e
  df ar = df_mul_f(a, r);
  const float e = __fsub_rn(__fsub_rn(1.0f, ar.hi), ar.lo);
  return fast_two_sum(r, __fmul_rn(r, e));
}

// ------------------------------------------------------------------ elementary functions
// sqrt(a): the FP32 root r refined by one Newton step, r + (a - r^2) / (2 r), with a - r^2
// formed exactly (TwoProduct); ~1e-14 relative. a >= 0.
__device__ __forceinline__ df df_sqrt(df a) {
  if (!(a.hi > 0.0f)) return {0.0f, 0.0f};
  const float r = __fsqrt_rn(a.hi);
  const df rr = two_prod(r, r);
  const float e = __fadd_rn(__fsub_rn(__fsub_rn(a.hi, rr.hi), rr.lo), a.lo);
  return fast_two_sum(r, __fdiv_rn(e, __fmul_rn(2.0f, r)));
}

// Exact double-float of a Philox uniform w * 2^-32: the top 24 and the low 8 bits of w, then
// normalised (the low part below half an ulp of the high one; for w < 2^8 the high part is 0
// and the value moves into it, which df_sqrt and the products need).
__device__ __forceinline__ df df_u01(uint32_t w) {
  return fast_two_sum(__fmul_rn((float)(w & 0xffffff00u), 2.3283064365386963e-10f),
                      __fmul_rn((float)(w & 0xffu), 2.3283064365386963e-10f));
}

// sin(2 pi v) and cos(2 pi v) for any v of moderate size (|4 v| < 2^22), ~1e-14 absolute:
// v = q/4 + r with q = nearest integer to 4v, so x = 2 pi r lies in [-pi/4, pi/4] (r exact);
// sin x and cos x from their Taylor series in Horner form, the orders up to x^9 / x^8 in
// double-float, the smaller tail (below 3e-8 of the result) in FP32; the quadrant q mod 4
// then swaps and negates (sin(x + q pi/2), cos(x + q pi/2)).
__device__ __forceinline__ float4 df_sincos_2pi_inl(float vhi, float vlo) {
  const df v = {vhi, vlo};
  const float q = rintf(4.0f * v.hi);
  const df r = df_add_f(v, -0.25f * q);
  const df x = df_mul(r, df{6.2831855f, -1.7484555e-07f});
  const df x2 = df_mul(x, x);
  const float t = x2.hi;
  // sin x / x = 1 - x2/3! + x2^2/5! - x2^3/7! + x2^4/9! - x2^5/11! + x2^6/13! - x2^7/15!
  const float st = t * (-2.5052108e-08f + t * (1.6059044e-10f - t * 7.6471636e-13f));
  df ps = df_add_f(df{2.7557319e-06f, 3.7935712e-14f}, st);
  ps = df_add(df_mul(x2, ps), df{-0.0001984127f, 2.7255969e-12f});
  ps = df_add(df_mul(x2, ps), df{0.008333334f, -4.346172e-10f});
  ps = df_add(df_mul(x2, ps), df{-0.16666667f, 4.967054e-09f});
  ps = df_add_f(df_mul(x2, ps), 1.0f);
  const df sx = df_mul(x, ps);
  // cos x = 1 - x2/2! + x2^2/4! - x2^3/6! + x2^4/8! - x2^5/10! + x2^6/12! - x2^7/14! + x2^8/16!
  const float ct = t * (-2.755732e-07f + t * (2.0876756e-09f + t * (-1.1470745e-11f + t * 4.7794773e-14f)));
  df pc = df_add_f(df{2.4801588e-05f, -3.406996e-13f}, ct);
  pc = df_add(df_mul(x2, pc), df{-0.0013888889f, 3.3631094e-11f});
  pc = df_add(df_mul(x2, pc), df{0.041666668f, -1.2417635e-09f});
  pc = df_add_f(df_mul(x2, pc), -0.5f);
  pc = df_add_f(df_mul(x2, pc), 1.0f);
  const int quad = ((int)q) & 3;
  const df ns = {-sx.hi, -sx.lo}, nc = {-pc.hi, -pc.lo};
  const df s = quad == 0 ? sx : (quad == 1 ? pc : (quad == 2 ? ns : nc));
  const df c = quad == 0 ? pc : (quad == 1 ? ns : (quad == 2 ? nc : sx));
  return make_float4(s.hi, s.lo, c.hi, c.lo);
}

// The same out of line (one copy per kernel for the orientation, rotation and eik call
// sites: these run once per move on few lanes, where instruction fetch, not arithmetic,
// sets the time), the result returned in registers.
static __device__ __noinline__ float4 df_sincos_2pi_out(float vhi, float vlo) { return df_sincos_2pi_inl(vhi, vlo); }

__device__ __forceinline__ void df_sincos_2pi(df v, df& s, df& c) {
  const float4 r = df_sincos_2pi_out(v.hi, v.lo);
  s = df{r.x, r.y};
  c = df{r.z, r.w};
}

// q e^{i 2 pi k f} as double-float complex {re hi, re lo, im hi, im lo}, straight from the sine
// and cosine of k f: every entry of the eik tables is independent, so a move's rows are one
// evaluation deep instead of a chain of kmax complex products on few lanes.
__device__ __forceinline__ float4 df_eik(double f, int k, df q) {
  df sn, cs;
  df_sincos_2pi(df_mul_f(df_from(f), (float)k), sn, cs);
  const df r = df_mul(q, cs), i = df_mul(q, sn);
  return make_float4(r.hi, r.lo, i.hi, i.lo);
}

// The quaternion of Rotate_Quaternions (mc_utilities.h:423-457, uniform rotation from three
// uniforms) with the uniforms given as Philox words, in double-float on the FP32 pipe, to ~1e-13
// relative. Half 0: (q0, q1) from u and v, half 1: (q2, q3) from u and w.
__device__ __forceinline__ float4 df_quaternion_half(uint32_t wu, uint32_t wangle, int half) {
  const df u = df_u01(wu);
  df s, c;
  df_sincos_2pi(df_u01(wangle), s, c);
  const df m = df_sqrt(half ? u : df_add_f(df{-u.hi, -u.lo}, 1.0f));
  const df a = df_mul(m, s), b = df_mul(m, c);
  return make_float4(a.hi, a.lo, b.hi, b.lo);
}

// Component d of (x, y, z) rotated by the quaternion halves q[0], q[1]. With (i, j, k) the axes
// d, d+1, d+2 and e the vector part, row d of the matrix is 1 - 2 (e_j^2 + e_k^2) at i,
// 2 (e_i e_j - q0 e_k) at j and 2 (e_i e_k + q0 e_j) at k.
__device__ __forceinline__ df df_rotated(float4 qa, float4 qb, int d, df x, df y, df z) {
  const df q0 = {qa.x, qa.y}, q1 = {qa.z, qa.w}, q2 = {qb.x, qb.y}, q3 = {qb.z, qb.w};
  auto pick3 = [d](df a, df b, df c) { return d == 0 ? a : (d == 1 ? b : c); };
  const df ei = pick3(q1, q2, q3), ej = pick3(q2, q3, q1), ek = pick3(q3, q1, q2);
  auto two = [](df p) { return df{2.0f * p.hi, 2.0f * p.lo}; };
  auto neg = [](df p) { return df{-p.hi, -p.lo}; };
  const df ti = df_mul(pick3(x, y, z), df_add_f(neg(two(df_add(df_mul(ej, ej), df_mul(ek, ek)))), 1.0f));
  const df tj = df_mul(pick3(y, z, x), two(df_add(df_mul(ei, ej), neg(df_mul(q0, ek)))));
  const df tk = df_mul(pick3(z, x, y), two(df_add(df_mul(ei, ek), df_mul(q0, ej))));
  return df_add(df_add(pick3(ti, tk, tj), pick3(tj, ti, tk)), pick3(tk, tj, ti));  // x, y, z terms in turn
}

__device__ __forceinline__ void df_rotate_quaternion(double& x, double& y, double& z, uint32_t wu, uint32_t wv,
                                                     uint32_t ww) {
  const float4 qa = df_quaternion_half(wu, wv, 0), qb = df_quaternion_half(wu, ww, 1);
  const df X = df_from(x), Y = df_from(y), Z = df_from(z);
  x = df_to(df_rotated(qa, qb, 0, X, Y, Z));
  y = df_to(df_rotated(qa, qb, 1, X, Y, Z));
  z = df_to(df_rotated(qa, qb, 2, X, Y, Z));
}

}  // namespace grx
