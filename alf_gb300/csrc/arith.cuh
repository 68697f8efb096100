#pragma once
#include "common.cuh"
#include "dfloat.cuh"

// |x| well inside the normal range (2^-900 .. 2^900), x / 2 and -x, on the integer pipes.
ALF_DEV bool alf_normal(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ff;
  return e - 123u < 1800u;
}
ALF_DEV double alf_half(double x) { return __hiloint2double(__double2hiint(x) - (1 << 20), __double2loint(x)); }
ALF_DEV double alf_flip(double x) { return __hiloint2double(__double2hiint(x) ^ (int)0x80000000u, __double2loint(x)); }
// 1/y without a division, for arguments in alf_normal's range: Chebyshev's method (third order: J. F. Traub,
// Iterative Methods for the Solution of Equations, 1964), x - u - u^2 f''/(2 f') with u = f/f', once for
// f(x) = 1/x - y from PTX's gross approximation r: with e = 1 - y r, r (1 + e + e^2), off by e^3 of the
// result.  The approximation sees the upper word of its argument alone (20 bits of mantissa): over
// all of these |e| <= 2^-19.9, so the result is off by 0.51 ulp at most.  CUDA's reciprocal in its
// place: 4 x 4 FP64 sweeps 4.69 -> 4.77 ms, 16 x 16 53.1 -> 54.1.
ALF_DEV double alf_rcp_seed(double y) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(y));
  return r;
}
ALF_DEV double alf_rcp_n(double y) {
  const double r = alf_rcp_seed(y), e = fma(-y, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
// sqrt(t) given r = 1/sqrt(t): one Newton step for s^2 = t from t r, its slope 2 s from r (0.5 ulp).
ALF_DEV double alf_sqrt_n(double t, double r) {
  const double s = t * r;
  return fma(fma(-s, s, t), alf_half(r), s);
}
// 1/y: seven dependent FP64 instructions fewer than a division.
ALF_DEV double alf_rcp(double y) { return alf_normal(y) ? alf_rcp_n(y) : 1.0 / y; }

// Scalar arithmetic shared by the update and QR kernels.  ArD: FP64 complex (the
// plain form: ratios must agree with an FP64 reference to ~1e-10 even where
// 1 + Delta (1 - G_jj) cancels).  ArF: double-float on the FP32 pipes (the mixed
// form; dfloat.cuh).  Z is a complex value, R a real one; both types are 16 and
// 8 bytes in either arithmetic, so shared-memory layouts do not change.
struct ArD {
  typedef zd Z;
  typedef double R;
  static constexpr bool kDoubleFloat = false, kReal = false;
  static ALF_DEV Z mk(zd a) { return a; }
  typedef zd S;  // element of a matrix held in this arithmetic in memory
  static ALF_DEV Z ld(S a) { return a; }
  static ALF_DEV Z inv(Z a) { return zinv(a); }
  static ALF_DEV zd wide(Z a) { return a; }
  static ALF_DEV R mkr(double a) { return a; }
  static ALF_DEV Z one() { return zmk(1.0, 0.0); }
  static ALF_DEV Z zero() { return zmk(0.0, 0.0); }
  static ALF_DEV Z mul(Z a, Z b) { return zmul(a, b); }
  static ALF_DEV Z sub(Z a, Z b) { return zsub(a, b); }
  static ALF_DEV Z add(Z a, Z b) { return zadd(a, b); }
  static ALF_DEV Z neg(Z a) { return zmk(-a.x, -a.y); }
  static ALF_DEV Z mac(Z c, Z a, Z b) { return zfma(a, b, c); }
  static ALF_DEV Z scale(Z a, R s) { return zscale(a, s); }
  static ALF_DEV R re(Z a) { return a.x; }
  static ALF_DEV R mulr(R a, R b) { return a * b; }
  static ALF_DEV bool gt(R a, R b) { return a > b; }
  static ALF_DEV Z rcp(Z a) {
    const double s = alf_rcp(a.x * a.x + a.y * a.y);
    return zmk(a.x * s, -a.y * s);
  }
  static ALF_DEV zd unit(Z a) { const double r = sqrt(a.x * a.x + a.y * a.y); return zmk(a.x / r, a.y / r); }
  static ALF_DEV Z shfl(Z a, int src) {
    return zmk(__shfl_sync(0xffffffffu, a.x, src), __shfl_sync(0xffffffffu, a.y, src));
  }
  static ALF_DEV Z shfl_xor(Z a, int o) {
    return zmk(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
  }
  static ALF_DEV Z conj(Z a) { return zmk(a.x, -a.y); }
  static ALF_DEV Z mkz(R r, R i) { return zmk(r, i); }
  static ALF_DEV R im(Z a) { return a.y; }
  static ALF_DEV R abs2(Z a) { return a.x * a.x + a.y * a.y; }
  static ALF_DEV R abs2add(Z a, R s) { return fma(a.x, a.x, fma(a.y, a.y, s)); }
  static ALF_DEV R abs2sub(R s, Z a) { return fma(-a.x, a.x, fma(-a.y, a.y, s)); }
  static ALF_DEV R rzero() { return 0.0; }
  static ALF_DEV R radd(R a, R b) { return a + b; }
  static ALF_DEV R rsub(R a, R b) { return a - b; }
  static ALF_DEV R rneg(R a) { return -a; }
  static ALF_DEV R rsqrt_(R a) { return sqrt(a); }
  static ALF_DEV R rrcp(R a) { return alf_rcp(a); }
  static ALF_DEV R rmax0(R a) { return a > 0.0 ? a : 0.0; }
  static ALF_DEV bool rzero_p(R a) { return a == 0.0; }
  static ALF_DEV bool rneg_p(R a) { return a < 0.0; }
  static ALF_DEV double rwide(R a) { return a; }
  static ALF_DEV R rcopysign(R mag, R sgn) { return copysign(mag, sgn); }
  static ALF_DEV R rshfl_xor(R a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
};
struct ArF {
  typedef dfz Z;
  typedef dff R;
  static constexpr bool kDoubleFloat = true, kReal = false;
  static ALF_DEV Z mk(zd a) { return dz_make(a); }
  typedef dfz S;
  static ALF_DEV Z ld(S a) { return a; }
  static ALF_DEV zd wide(Z a) { return dz_wide(a); }
  static ALF_DEV R mkr(double a) { return df_make(a); }
  static ALF_DEV Z one() { return dfz{{1.f, 0.f}, {0.f, 0.f}}; }
  static ALF_DEV Z zero() { return dfz{{0.f, 0.f}, {0.f, 0.f}}; }
  static ALF_DEV Z mul(Z a, Z b) { return dz_mul(a, b); }
  static ALF_DEV Z sub(Z a, Z b) { return dz_sub(a, b); }
  static ALF_DEV Z add(Z a, Z b) { return dz_add(a, b); }
  static ALF_DEV Z neg(Z a) { return dfz{df_neg(a.r), df_neg(a.i)}; }
  static ALF_DEV Z mac(Z c, Z a, Z b) { return dz_mac(c, a, b); }
  static ALF_DEV Z scale(Z a, R s) { return dz_scale(a, s); }
  static ALF_DEV R re(Z a) { return a.r; }
  static ALF_DEV R mulr(R a, R b) { return df_mul(a, b); }
  static ALF_DEV bool gt(R a, R b) { return df_gt(a, b); }
  static ALF_DEV Z rcp(Z a) { return dz_rcp(a); }
  static ALF_DEV zd unit(Z a) { return dz_wide(dz_unit(a)); }
  static ALF_DEV Z shfl(Z a, int src) {
    Z r;
    r.r.h = __shfl_sync(0xffffffffu, a.r.h, src); r.r.l = __shfl_sync(0xffffffffu, a.r.l, src);
    r.i.h = __shfl_sync(0xffffffffu, a.i.h, src); r.i.l = __shfl_sync(0xffffffffu, a.i.l, src);
    return r;
  }
  static ALF_DEV Z shfl_xor(Z a, int o) {
    Z r;
    r.r.h = __shfl_xor_sync(0xffffffffu, a.r.h, o); r.r.l = __shfl_xor_sync(0xffffffffu, a.r.l, o);
    r.i.h = __shfl_xor_sync(0xffffffffu, a.i.h, o); r.i.l = __shfl_xor_sync(0xffffffffu, a.i.l, o);
    return r;
  }
  static ALF_DEV Z conj(Z a) { return dz_conj(a); }
  static ALF_DEV Z mkz(R r, R i) { return dfz{r, i}; }
  static ALF_DEV R im(Z a) { return a.i; }
  static ALF_DEV R abs2(Z a) { return dz_abs2(a); }
  static ALF_DEV R rzero() { return dff{0.f, 0.f}; }
  static ALF_DEV R radd(R a, R b) { return df_add(a, b); }
  static ALF_DEV R rsub(R a, R b) { return df_sub(a, b); }
  static ALF_DEV R rneg(R a) { return df_neg(a); }
  static ALF_DEV R rsqrt_(R a) { return df_sqrt(a); }
  static ALF_DEV R rrcp(R a) { return df_rcp(a); }
  static ALF_DEV R rmax0(R a) { return a.h > 0.f ? a : dff{0.f, 0.f}; }
  static ALF_DEV bool rzero_p(R a) { return a.h == 0.f && a.l == 0.f; }
  static ALF_DEV bool rneg_p(R a) { return a.h < 0.f; }
  static ALF_DEV double rwide(R a) { return df_wide(a); }
  static ALF_DEV R rcopysign(R mag, R sgn) { return ((mag.h < 0.f) != (sgn.h < 0.f)) ? df_neg(mag) : mag; }
  static ALF_DEV R rshfl_xor(R a, int o) {
    return dff{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)};
  }
};

// Real FP64: the plain form on models whose vertex exponentials and transition factors are all
// real (the hopping exponentials always are).  Every matrix of the sweep then has zero imaginary
// parts, and ArD's complex products spend three of four FP64 instructions on them; the real
// parts come out of the same operations in the same order.  Matrices stay complex128 in memory
// (mk takes the real part, wide writes a zero imaginary part).
struct ArRe {
  typedef double Z;
  typedef double R;
  static constexpr bool kDoubleFloat = false, kReal = true;
  static ALF_DEV Z mk(zd a) { return a.x; }
  typedef zd S;
  static ALF_DEV Z ld(S a) { return a.x; }
  static ALF_DEV Z inv(Z a) { return 1.0 / a; }
  static ALF_DEV zd wide(Z a) { return zmk(a, 0.0); }
  static ALF_DEV R mkr(double a) { return a; }
  static ALF_DEV Z one() { return 1.0; }
  static ALF_DEV Z zero() { return 0.0; }
  static ALF_DEV Z mul(Z a, Z b) { return a * b; }
  static ALF_DEV Z sub(Z a, Z b) { return a - b; }
  static ALF_DEV Z add(Z a, Z b) { return a + b; }
  static ALF_DEV Z neg(Z a) { return -a; }
  static ALF_DEV Z mac(Z c, Z a, Z b) { return fma(a, b, c); }
  static ALF_DEV Z scale(Z a, R s) { return a * s; }
  static ALF_DEV R re(Z a) { return a; }
  static ALF_DEV R im(Z) { return 0.0; }
  static ALF_DEV R mulr(R a, R b) { return a * b; }
  static ALF_DEV bool gt(R a, R b) { return a > b; }
  static ALF_DEV Z rcp(Z a) { return alf_rcp(a); }
  static ALF_DEV Z shfl(Z a, int src) { return __shfl_sync(0xffffffffu, a, src); }
  static ALF_DEV Z shfl_xor(Z a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
  static ALF_DEV Z conj(Z a) { return a; }
  static ALF_DEV Z mkz(R r, R) { return r; }
  static ALF_DEV R abs2(Z a) { return a * a; }
  static ALF_DEV R abs2add(Z a, R s) { return fma(a, a, s); }
  static ALF_DEV R abs2sub(R s, Z a) { return fma(-a, a, s); }
  static ALF_DEV R rzero() { return 0.0; }
  static ALF_DEV R radd(R a, R b) { return a + b; }
  static ALF_DEV R rsub(R a, R b) { return a - b; }
  static ALF_DEV R rneg(R a) { return -a; }
  static ALF_DEV R rsqrt_(R a) { return sqrt(a); }
  static ALF_DEV R rrcp(R a) { return alf_rcp(a); }
  static ALF_DEV R rmax0(R a) { return a > 0.0 ? a : 0.0; }
  static ALF_DEV bool rzero_p(R a) { return a == 0.0; }
  static ALF_DEV bool rneg_p(R a) { return a < 0.0; }
  static ALF_DEV double rwide(R a) { return a; }
  static ALF_DEV R rcopysign(R mag, R sgn) { return copysign(mag, sgn); }
  static ALF_DEV R rshfl_xor(R a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
};

// Real double-float: ArF on real models (the visits and flush operands of the mixed form).
struct ArFRe {
  typedef dff Z;
  typedef dff R;
  static constexpr bool kDoubleFloat = true, kReal = true;
  static ALF_DEV Z mk(zd a) { return df_make(a.x); }
  static ALF_DEV zd wide(Z a) { return zmk(df_wide(a), 0.0); }
  static ALF_DEV Z one() { return dff{1.f, 0.f}; }
  static ALF_DEV Z zero() { return dff{0.f, 0.f}; }
  static ALF_DEV Z mul(Z a, Z b) { return df_mul(a, b); }
  static ALF_DEV Z sub(Z a, Z b) { return df_sub(a, b); }
  static ALF_DEV Z add(Z a, Z b) { return df_add(a, b); }
  static ALF_DEV Z neg(Z a) { return df_neg(a); }
  static ALF_DEV Z mac(Z c, Z a, Z b) { return df_fma(c, a, b); }
  static ALF_DEV Z rcp(Z a) { return df_rcp(a); }
  static ALF_DEV Z shfl(Z a, int src) {
    return dff{__shfl_sync(0xffffffffu, a.h, src), __shfl_sync(0xffffffffu, a.l, src)};
  }
};
