// Arithmetic of the bond splits' inner loops, QA<T>: T = double (complex128
// form) or ff (double-float on the FP32 pipe, mixed form).
//
//   E  element of the working matrix (16 bytes in both forms)
//   S  real accumulator / scalar (8 bytes in both forms)
//
// Accumulators run unnormalised inside a loop and across a group's lanes
// (dotj, abs2_acc, group_sum); fin() normalises them.
#pragma once

#include "common.cuh"
#include "ff.cuh"

namespace otb {

template <typename T>
struct QA;

// FP32 estimates without denormal handling (half the latency of the library
// forms): a denormal argument counts as zero, so callers keep to normal ones
__device__ __forceinline__ float rsqrt_est(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_est(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// FP64 -> FP32 by integer instructions: a conversion takes the FP64 pipe like
// any FP64 instruction.  Truncated (*rest: the cut bits); values below 2^-126
// are 0, those above the range infinite or NaN.
__device__ __forceinline__ float trunc32(double d, unsigned* rest = nullptr) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned e = (hi >> 20) & 0x7ffu;
  const unsigned f =
      (hi & 0x80000000u) | (min(e - 896u, 255u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
  const bool normal = e > 896u;
  if (rest) *rest = normal ? lo & 0x1fffffffu : 0u;
  return __uint_as_float(normal ? f : 0u);
}
__device__ __forceinline__ cx<float> trunc32(const cx<double>& a) { return mk<float>(trunc32(a.x), trunc32(a.y)); }

constexpr float FP32_NORMAL = 1.17549435e-38f;   // smallest normal number

template <>
struct QA<double> {
  typedef cx<double> E;
  typedef double S;
  static constexpr bool kFF = false;
  // A unitary rotation of two columns by the complex tangent tau (FP32, so
  // exact in both arithmetics): u <- c (u - conj(tau) v), v <- c (v + tau u),
  // c = 1 / sqrt(1 + |tau|^2).
  struct Rot {
    double tx, ty, c;
  };
  static __device__ __forceinline__ E from(cx<double> z) { return z; }
  static __device__ __forceinline__ cx<double> to(const E& e) { return e; }
  static __device__ __forceinline__ S zero() { return 0.0; }
  static __device__ __forceinline__ E zeroE() { return mk<double>(0.0, 0.0); }
  static __device__ __forceinline__ E realE(S s) { return mk<double>(s, 0.0); }
  static __device__ __forceinline__ float tof(S s) { return (float)s; }
  static __device__ __forceinline__ double tod(S s) { return s; }
  static __device__ __forceinline__ S fin(S v) { return v; }
  template <int G>
  static __device__ __forceinline__ S group_sum(S v) {
#pragma unroll
    for (int off = G >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off, 32);
    return v;
  }
  static __device__ __forceinline__ S abs2_acc(const E& x, S acc) { return fma(x.x, x.x, fma(x.y, x.y, acc)); }
  static __device__ __forceinline__ float abs2_32(const E& x, float acc) {
    const cx<float> y = trunc32(x);
    return fmaf(y.x, y.x, fmaf(y.y, y.y, acc));
  }
  // (wr, wi) += conj(a) x
  static __device__ __forceinline__ void dotj(S& wr, S& wi, const E& a, const E& x) {
    wr = fma(a.x, x.x, fma(a.y, x.y, wr));
    wi = fma(a.x, x.y, fma(-a.y, x.x, wi));
  }
  // x - a (bx + i by)
  static __device__ __forceinline__ E sub_scaled(const E& x, const E& a, S bx, S by) {
    return mk<double>(fma(a.y, by, fma(-a.x, bx, x.x)), fma(-a.y, bx, fma(-a.x, by, x.y)));
  }
  static __device__ __forceinline__ S mul(S a, S b) { return a * b; }
  static __device__ __forceinline__ E scaleE(const E& a, S s) { return mk<double>(a.x * s, a.y * s); }
  static __device__ __forceinline__ E conj_scale(const E& a, S s) { return mk<double>(a.x * s, -a.y * s); }
  // powers of two: of the largest magnitude in an unsigned key, and x 2^e
  typedef double P;
  static __device__ __forceinline__ unsigned mag_key(const E& a) {
    return max((unsigned)__double2hiint(a.x) & 0x7fffffffu, (unsigned)__double2hiint(a.y) & 0x7fffffffu);
  }
  static __device__ __forceinline__ int key_exponent(unsigned key) {
    const int e = (int)(key >> 20);
    return (e == 0 || e == 0x7ff) ? 0 : e - 1023;
  }
  static __device__ __forceinline__ P pow2(int e) { return ldexp(1.0, e); }
  static __device__ __forceinline__ E ldexpE(const E& a, P p2) { return mk<double>(a.x * p2, a.y * p2); }
  static __device__ __forceinline__ E conj(const E& a) { return mk<double>(a.x, -a.y); }
  static __device__ __forceinline__ E add(const E& a, const E& b) { return a + b; }
  static __device__ __forceinline__ S fromd(double d) { return d; }
  // complex multiply-accumulate of the contractions
  typedef cx<double> Acc;
  static __device__ __forceinline__ Acc acc_zero() { return mk<double>(0.0, 0.0); }
  static __device__ __forceinline__ void acc_fma(Acc& f, const E& a, const E& b) { cfma(f, a, b); }
  static __device__ __forceinline__ void acc_fmaj(Acc& f, const E& a, const E& b) { cjfma(f, a, b); }
  static __device__ __forceinline__ E acc_value(const Acc& f) { return f; }
  // 1 / sqrt(u), 0 for u <= 0: the FP32 estimate y with the first two terms of
  // the binomial series of (1 - r)^-1/2, r = 1 - u y^2, in FP64 (what is left out
  // is below 2^-64 before the final rounding), five FP64 instructions instead of
  // the library's square root and division.  Values below FP32's normal range
  // are scaled into it, those below 2^-326 count as zero.
  static __device__ __forceinline__ S rsqrt(S u) {
    if ((float)u < FP32_NORMAL && u > 0.0) return 0x1p+100 * rsqrt_normal(u * 0x1p+200);
    return rsqrt_normal(u);
  }
  static __device__ __forceinline__ S rsqrt_normal(S u) {
    const float uf = (float)u;
    if (!(uf >= FP32_NORMAL)) return u * 0.0;   // 0 (NaN stays NaN)
    const double y = (double)rsqrt_est(uf);
    const double r = fma(-u, y * y, 1.0);
    return fma(y * r, fma(0.375, r, 0.5), y);
  }
  // (x, y) = (gr, gi) rr summed over a pair's G lanes, in FP32; rr is about
  // 1 / (|u| |v|)
  template <int G>
  static __device__ __forceinline__ void gamma(S gr, S gi, float rr, float& x, float& y) {
    const bool up = threadIdx.x & (G >> 1);
    const float v = (float)(half_sum<G>(gr, gi) * (double)rr);
    const float o = __shfl_xor_sync(0xffffffffu, v, G >> 1, 32);
    x = up ? o : v;
    y = up ? v : o;
  }
  // The sum of a over the G lanes in the group's lower half, of b in its upper
  // half: the halves swap what they do not keep first, so that the two sums
  // take log2 G additions, not 2 log2 G.
  template <int G>
  static __device__ __forceinline__ S half_sum(S a, S b) {
    const bool up = threadIdx.x & (G >> 1);
    S v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, G >> 1, 32);
#pragma unroll
    for (int off = G >> 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off, 32);
    return v;
  }
  // (wr, wi) summed over a group's G lanes (the third argument, about 1 over a
  // bound of the sums, steers the double-float form)
  template <int G>
  static __device__ __forceinline__ void dot_sum(S& wr, S& wi, float) {
    const bool up = threadIdx.x & (G >> 1);
    const S v = half_sum<G>(wr, wi);
    const S o = __shfl_xor_sync(0xffffffffu, v, G >> 1, 32);
    wr = up ? o : v;
    wi = up ? v : o;
  }
  static __device__ __forceinline__ float diff(S a, S b) { return (float)(a - b); }
  static __device__ __forceinline__ S shift(S a, float d) { return a + (double)d; }
  static __device__ __forceinline__ Rot rotation(float tx, float ty) {
    Rot q;
    q.tx = (double)tx;
    q.ty = (double)ty;
    q.c = rsqrt_normal(fma(q.tx, q.tx, fma(q.ty, q.ty, 1.0)));
    return q;
  }
  static __device__ __forceinline__ void rotate(const Rot& q, E& u, E& v) {
    const double nux = fma(-q.tx, v.x, fma(-q.ty, v.y, u.x)), nuy = fma(-q.tx, v.y, fma(q.ty, v.x, u.y));
    const double nvx = fma(q.tx, u.x, fma(-q.ty, u.y, v.x)), nvy = fma(q.tx, u.y, fma(q.ty, u.x, v.y));
    u = mk<double>(q.c * nux, q.c * nuy);
    v = mk<double>(q.c * nvx, q.c * nvy);
  }
  static __device__ __forceinline__ float jacobi_tol(int m) { return sqrtf((float)m) * 1.1102230246251565e-16f; }
  static __device__ __forceinline__ float jacobi_floor(int m) { return 16.f * sqrtf((float)m) * 1.1102230246251565e-16f; }
};

template <>
struct QA<ff> {
  typedef cff E;
  typedef ff S;
  static constexpr bool kFF = true;
  struct Rot {
    float tx, ty;
    ff c;
  };
  static __device__ __forceinline__ E from(cx<double> z) { return cff_from(z); }
  static __device__ __forceinline__ cx<double> to(const E& e) { return cff_to(e); }
  static __device__ __forceinline__ S zero() { return ff_make(0.f, 0.f); }
  static __device__ __forceinline__ E realE(S s) {
    E r;
    r.x = s;
    r.y = zero();
    return r;
  }
  static __device__ __forceinline__ E zeroE() { return realE(zero()); }
  static __device__ __forceinline__ float tof(S s) { return s.hi; }
  static __device__ __forceinline__ double tod(S s) { return ff_to(s); }
  static __device__ __forceinline__ S fin(S v) { return ffacc_norm(v.hi, v.lo); }
  // the high words through an error-free sum, everything else in the low word
  template <int G>
  static __device__ __forceinline__ S group_sum(S v) {
#pragma unroll
    for (int off = G >> 1; off > 0; off >>= 1) {
      const ff o = ff_shfl_xor(v, off);
      const ff s = two_sum(v.hi, o.hi);
      v = ff_make(s.hi, __fadd_rn(__fadd_rn(v.lo, o.lo), s.lo));
    }
    return v;
  }
  static __device__ __forceinline__ float abs2_32(const E& x, float acc) {
    return fmaf(x.x.hi, x.x.hi, fmaf(x.y.hi, x.y.hi, acc));
  }
  static __device__ __forceinline__ S abs2_acc(const E& x, S acc) {
    ffp_acc(x.x.hi, x.x.lo, x.x.hi, x.x.lo, acc.hi, acc.lo);
    ffp_acc(x.y.hi, x.y.lo, x.y.hi, x.y.lo, acc.hi, acc.lo);
    return acc;
  }
  // wr + i wi += conj(a) x as compensated accumulators
  static __device__ __forceinline__ void dotj(S& wr, S& wi, const E& a, const E& x) {
    ffp_acc(a.x.hi, a.x.lo, x.x.hi, x.x.lo, wr.hi, wr.lo);
    ffp_acc(a.x.hi, a.x.lo, x.y.hi, x.y.lo, wi.hi, wi.lo);
    ffp_acc(a.y.hi, a.y.lo, x.y.hi, x.y.lo, wr.hi, wr.lo);
    ffp_acc(-a.y.hi, -a.y.lo, x.x.hi, x.x.lo, wi.hi, wi.lo);
  }
  // x - a (bx + i by), each component one compensated accumulation
  static __device__ __forceinline__ E sub_scaled(const E& x, const E& a, S bx, S by) {
    E r;
    float h = x.x.hi, l = x.x.lo;
    ffp_acc(-a.x.hi, -a.x.lo, bx.hi, bx.lo, h, l);
    ffp_acc(a.y.hi, a.y.lo, by.hi, by.lo, h, l);
    r.x = ffacc_norm(h, l);
    h = x.y.hi;
    l = x.y.lo;
    ffp_acc(-a.x.hi, -a.x.lo, by.hi, by.lo, h, l);
    ffp_acc(-a.y.hi, -a.y.lo, bx.hi, bx.lo, h, l);
    r.y = ffacc_norm(h, l);
    return r;
  }
  static __device__ __forceinline__ S mul(S a, S b) { return ff_mul(a, b); }
  static __device__ __forceinline__ E scaleE(const E& a, S s) { return cff_scale(a, s); }
  static __device__ __forceinline__ E conj_scale(const E& a, S s) { return cff_conj(cff_scale(a, s)); }
  typedef float P;
  static __device__ __forceinline__ unsigned mag_key(const E& a) {
    return max(__float_as_uint(a.x.hi) & 0x7fffffffu, __float_as_uint(a.y.hi) & 0x7fffffffu);
  }
  static __device__ __forceinline__ int key_exponent(unsigned key) {
    const int e = (int)(key >> 23);
    return (e == 0 || e == 0xff) ? 0 : e - 127;
  }
  static __device__ __forceinline__ P pow2(int e) { return ldexpf(1.f, e); }
  static __device__ __forceinline__ E ldexpE(const E& a, P p2) { return cff_ldexp(a, p2); }
  static __device__ __forceinline__ E conj(const E& a) { return cff_conj(a); }
  static __device__ __forceinline__ E add(const E& a, const E& b) { return cff_add(a, b); }
  static __device__ __forceinline__ S fromd(double d) { return ff_from(d); }
  typedef ccacc Acc;
  static __device__ __forceinline__ Acc acc_zero() { return ccacc_zero(); }
  static __device__ __forceinline__ void acc_fma(Acc& f, const E& a, const E& b) { ccacc_fma(f, a, b); }
  static __device__ __forceinline__ void acc_fmaj(Acc& f, const E& a, const E& b) { ccacc_fmaj(f, a, b); }
  static __device__ __forceinline__ E acc_value(const Acc& f) { return ccacc_cff(f); }
  // 1 / sqrt(u), 0 for u <= 0: as in FP64, the residual 1 - u y^2 formed from
  // exact products.  A squared norm below the normal range has no digits left
  // and counts as zero (a column 1e-19 of the largest, 2^-48 being rounding).
  static __device__ __forceinline__ S rsqrt(S u) {
    if (!(u.hi >= FP32_NORMAL)) return ff_make(u.hi * 0.f, 0.f);
    const float y = rsqrt_est(u.hi);
    const float p = __fmul_rn(y, y), pe = __fmaf_rn(y, y, -p);
    float r = __fmaf_rn(-u.hi, p, 1.f);
    r = __fmaf_rn(-u.hi, pe, r);
    r = __fmaf_rn(-u.lo, p, r);
    return fast_two_sum(y, __fmul_rn(y, __fmul_rn(r, __fmaf_rn(0.375f, r, 0.5f))));
  }
  // The sum over a group's G lanes (4 <= G <= 32) of a in the group's lower
  // half and of b in its upper half (the halves swap what they do not keep
  // first), for values whose lanes' magnitudes add up to at most a known bound,
  // r ~ 1 / bound.  Every lane's high word is split at two fixed grids, 2^-22
  // and 2^-41 of the bound: the grid parts are integers whose sums stay below
  // 2^24 and add exactly in plain FP32, and what is left below them (with the
  // low word) is summed in FP32, 2^-48 of the bound.  Three shuffles and adds
  // per level, where a pair of error-free additions takes four shuffles and a
  // chain of six dependent adds (about 45 against 150 clocks a level).
  struct Parts {
    float p0, p1, p2;   // first grid, second grid, rest; in units of 1 / s
    float s;
  };
  template <int G>
  static __device__ __forceinline__ Parts half_sum(S a, S b, float r) {
    Parts g;
    g.s = __uint_as_float((__float_as_uint(r) & 0x7f800000u) + (22u << 23));
    const float c0 = 12582912.f, c1 = 24.f;   // 1.5 2^23 times the grids 1 and 2^-19
    const float a0 = __fsub_rn(__fmaf_rn(a.hi, g.s, c0), c0), b0 = __fsub_rn(__fmaf_rn(b.hi, g.s, c0), c0);
    const float ar = __fmaf_rn(a.hi, g.s, -a0), br = __fmaf_rn(b.hi, g.s, -b0);
    const float a1 = __fsub_rn(__fadd_rn(ar, c1), c1), b1 = __fsub_rn(__fadd_rn(br, c1), c1);
    const float a2 = __fmaf_rn(a.lo, g.s, __fsub_rn(ar, a1)), b2 = __fmaf_rn(b.lo, g.s, __fsub_rn(br, b1));
    const int h = G >> 1;
    const bool up = threadIdx.x & h;
    g.p0 = __fadd_rn(up ? b0 : a0, __shfl_xor_sync(0xffffffffu, up ? a0 : b0, h, 32));
    g.p1 = __fadd_rn(up ? b1 : a1, __shfl_xor_sync(0xffffffffu, up ? a1 : b1, h, 32));
    g.p2 = __fadd_rn(up ? b2 : a2, __shfl_xor_sync(0xffffffffu, up ? a2 : b2, h, 32));
#pragma unroll
    for (int off = h >> 1; off > 0; off >>= 1) {
      g.p0 = __fadd_rn(g.p0, __shfl_xor_sync(0xffffffffu, g.p0, off, 32));
      g.p1 = __fadd_rn(g.p1, __shfl_xor_sync(0xffffffffu, g.p1, off, 32));
      g.p2 = __fadd_rn(g.p2, __shfl_xor_sync(0xffffffffu, g.p2, off, 32));
    }
    return g;
  }
  // (x, y) = (gr, gi) r in FP32 (r ~ 1 / (|u| |v|) of a column pair)
  template <int G>
  static __device__ __forceinline__ void gamma(S gr, S gi, float r, float& x, float& y) {
    const bool up = threadIdx.x & (G >> 1);
    const Parts g = half_sum<G>(gr, gi, r);
    const float f = __uint_as_float((__float_as_uint(r) & 0x007fffffu) | ((127u - 22u) << 23));   // r / s
    const float v = f * (g.p0 + (g.p1 + g.p2));
    const float o = __shfl_xor_sync(0xffffffffu, v, G >> 1, 32);
    x = up ? o : v;
    y = up ? v : o;
  }
  template <int G>
  static __device__ __forceinline__ void dot_sum(S& wr, S& wi, float r) {
    const bool up = threadIdx.x & (G >> 1);
    const Parts g = half_sum<G>(wr, wi, r);
    const float is = __uint_as_float((254u << 23) - (__float_as_uint(g.s) & 0x7f800000u));   // 1 / s
    const ff v = sum3(g.p0, g.p1, g.p2, is);
    const ff o = ff_shfl_xor(v, G >> 1);
    wr = up ? o : v;
    wi = up ? v : o;
  }
  static __device__ __forceinline__ ff sum3(float a, float b, float c, float is) {
    const ff t = two_sum(a, b);
    const ff u = two_sum(t.hi, c);
    const ff v = fast_two_sum(u.hi, __fadd_rn(t.lo, u.lo));
    return ff_make(v.hi * is, v.lo * is);
  }
  static __device__ __forceinline__ float diff(S a, S b) {
    const ff s = two_sum(a.hi, -b.hi);
    return s.hi + (s.lo + (a.lo - b.lo));
  }
  static __device__ __forceinline__ S shift(S a, float d) {
    const ff s = two_sum(a.hi, d);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
  }
  static __device__ __forceinline__ Rot rotation(float tx, float ty) {
    Rot q;
    q.tx = tx;
    q.ty = ty;
    // 1 + |tau|^2 from exact squares (the larger first)
    const float a = __fmul_rn(tx, tx), ae = __fmaf_rn(tx, tx, -a);
    const float b = __fmul_rn(ty, ty), be = __fmaf_rn(ty, ty, -b);
    const ff m = fast_two_sum(fmaxf(a, b), fminf(a, b));
    const ff u = fast_two_sum(1.f, m.hi);
    q.c = rsqrt(ff_make(u.hi, __fadd_rn(u.lo, __fadd_rn(m.lo, __fadd_rn(ae, be)))));
    return q;
  }
  // (h, l) += a t for a double-float a and a float t
  static __device__ __forceinline__ void acc1(ff a, float t, float& h, float& l) {
    const float p = __fmul_rn(a.hi, t);
    const float e = __fmaf_rn(a.lo, t, __fmaf_rn(a.hi, t, -p));
    const ff s = two_sum(h, p);
    h = s.hi;
    l = __fadd_rn(l, __fadd_rn(s.lo, e));
  }
  static __device__ __forceinline__ ff comb(ff x, ff a, float ta, ff b, float tb, ff c) {
    float h = x.hi, l = x.lo;
    acc1(a, ta, h, l);
    acc1(b, tb, h, l);
    return ff_mul(fast_two_sum(h, l), c);
  }
  static __device__ __forceinline__ void rotate(const Rot& q, E& u, E& v) {
    E nu, nv;
    nu.x = comb(u.x, v.x, -q.tx, v.y, -q.ty, q.c);
    nu.y = comb(u.y, v.y, -q.tx, v.x, q.ty, q.c);
    nv.x = comb(v.x, u.x, q.tx, u.y, -q.ty, q.c);
    nv.y = comb(v.y, u.y, q.tx, u.x, q.ty, q.c);
    u = nu;
    v = nv;
  }
  // the unnormalised accumulations sit a few units above the 2^-48 unit
  // roundoff: stopping test at 4x and numerical-zero floor at 32x
  static __device__ __forceinline__ float jacobi_tol(int m) { return 4.f * sqrtf((float)m) * 3.6e-15f; }
  static __device__ __forceinline__ float jacobi_floor(int m) { return 32.f * sqrtf((float)m) * 3.6e-15f; }
};

}  // namespace otb
