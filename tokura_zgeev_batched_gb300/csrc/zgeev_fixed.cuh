// 64-bit fixed-point arithmetic for the eigenvalue path.
//
// GB300 issues about 2 FP64 multiply-adds per clock and SM, each with a
// latency of 64 clocks, but 32 32x32+64-bit integer multiply-adds (measured).
// A Hessenberg reduction and a QR iteration are chains of unitary
// transformations, under which no entry ever exceeds the matrix's Frobenius
// norm, so one exponent per matrix serves all of its entries and all steps:
// the matrix is held as 64-bit integers and every product of a coefficient
// (|c| <= 1) and an entry is formed from 32-bit halves with three integer
// multiply-adds, 5.4 times the rate of an FP64 one (1.6 to 3.7 times for whole calls).
//
// An entry x is V = round(x 2^p), ||V||_F in (2^60, 2^61), i.e. it is held
// to 2^-61 of the norm in absolute terms (FP64 holds each entry to 2^-53 of
// itself; an entry of a 64 x 64 matrix with entries of one size is about 2^-6
// of the norm). Rounding is therefore an absolute, normwise error, as in the
// backward error of the QR algorithm; matrices whose small entries mean more
// than that (graded and badly balanced ones: zgeev_fixed_guard.cuh) are left to the FP64 kernels. Against eigenvalues in
// extended precision the normwise errors are below the FP64 kernels' for the classes and orders measured (rms over
// ||A||_F, Gaussian entries: n = 4 2.2e-17 against 2.3e-16, n = 16 2.0e-17 against 1.9e-16, n = 64 4.5e-17 against
// 1.8e-16); relative errors of small eigenvalues are below or within four times theirs but for few (10 times for the smallest
// root of a polynomial whose constant term is 2^-8 to 2^-11 of the largest coefficient and stands in a column of its own).
//
// In memory and in registers an entry is S = V + 2^31 (zero is kZero): the
// signed halves that a product wants, V = 2^32 h + l, are S's high word and its
// low word less 2^31. Coefficients are scaled by 2^62 and split alike,
// C = Ch 2^32 + Cl, |Ch| <= 2^30, |Cl| <= 2^31. Then
//   V' = sum C V / 2^62 = 4 sum Ch h + (sum (Ch l + Cl h)) / 2^30
// (the products Cl l are left out: below a unit of V each, with either sign).
// The middle sum of a rotation's three products, c.re^2 + c.im^2 + s^2 = 1, is
// below sqrt(3) 2^61 + sqrt(3) 2^31 ||h||, so it fits 63 bits for ||V|| < 0.655 * 2^63.
// The QR works on H - sigma I, whose columns are below 2 ||A||_F (every shift is at
// most ||A||_F), and make_rotc takes entries below 2^62: ||V||_F <= 0.2495 * 2^63 at staging.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define TZG_HD __host__ __device__ __forceinline__
#else
#define TZG_HD inline
#endif

namespace tzg {

constexpr float kFixedNormMax = 0.2495f * 9223372036854775808.0f;  // bound of ||V||_F
constexpr long long kZero = 1LL << 31;
// Subdiagonals up to four units are negligible (2^-57 of the norm at most; LAPACK's own
// threshold is 2^-52 of the neighbouring diagonal entries).
constexpr long long kFixedSmall = 4;

struct cfx {  // complex entry
  long long x, y;
};
struct Limbs {  // h 2^32 + l, both signed
  int h, l;
};

// a b + c. As a multiplication and a sum: they become one instruction with 64-bit accumulation, where
// mad.wide becomes two and the C expression may be regrouped (a rotation: 53, 89 and 79 instructions).
TZG_HD long long mad_wide(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
  long long p;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(p) : "r"(a), "r"(b));
  asm("add.s64 %0, %1, %2;" : "=l"(p) : "l"(p), "l"(c));
  return p;
#else
  return (long long)a * b + c;
#endif
}
TZG_HD int high(long long v) { return (int)(v >> 32); }

// Halves of an entry, of a plain 64-bit value, and that value back.
TZG_HD Limbs entry_limbs(long long s) {
  Limbs r;
  r.h = (int)(s >> 32);
  r.l = (int)((unsigned)s ^ 0x80000000u);
  return r;
}
TZG_HD Limbs limbs(long long v) {
  Limbs r;
  r.l = (int)v;
  r.h = (int)(v >> 32) + (int)((unsigned)r.l >> 31);
  return r;
}
TZG_HD long long value(Limbs a) { return ((long long)a.h << 32) + a.l; }
TZG_HD Limbs negated(Limbs a) {  // for odd a.l (coefficients)
  Limbs r;
  r.h = -a.h;
  r.l = -a.l;
  return r;
}

TZG_HD int clz64(unsigned long long v) {  // 64 for 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
TZG_HD int clz32(unsigned v) {  // 32 for 0
#ifdef __CUDA_ARCH__
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}

// |v| or |v| - 1: enough for the position of the top bit.
TZG_HD unsigned long long mag64(long long v) { return (unsigned long long)(v ^ (v >> 63)); }
TZG_HD unsigned mag32(int v) { return (unsigned)(v ^ (v >> 31)); }

// Products and sums that are never contracted: every kernel computes the same shifts and decisions.
TZG_HD float mulf(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
TZG_HD float addf(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
TZG_HD float rsqrt_seed(float x) {  // x normal
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / sqrtf(x);
#endif
}
TZG_HD int float_to_int_sat(float x) {  // 2^31 - 1 above the range
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return x >= 2147483648.0f ? 2147483647 : (int)x;
#endif
}

// Starts of a rotation's sums (half a unit; 4 times the other is kZero), held in a register pair of their own
// (as literals they cost a move each time).
struct Starts {
  long long half, zero;
};
TZG_HD Starts make_starts(int one) { return Starts{(long long)one << 29, (long long)one << 29}; }

// 4 hh + mid / 2^30.
TZG_HD long long join(long long hh, long long mid) { return (hh << 2) + (mid >> 30); }

// One output of a rotation: c0 a + c1 b + c2 d as an entry.
TZG_HD long long dot3(const Starts& k, Limbs c0, Limbs a, Limbs c1, Limbs b, Limbs c2, Limbs d) {
  long long mid = mad_wide(c0.h, a.l, k.half);
  long long hh = mad_wide(c0.h, a.h, k.zero);
  mid = mad_wide(c1.h, b.l, mid);
  hh = mad_wide(c1.h, b.h, hh);
  mid = mad_wide(c2.h, d.l, mid);
  hh = mad_wide(c2.h, d.h, hh);
  mid = mad_wide(c0.l, a.h, mid);
  mid = mad_wide(c1.l, b.h, mid);
  mid = mad_wide(c2.l, d.h, mid);
  return join(hh, mid);
}

// 2^91 / sqrt(T) to a relative error of about 2^-57 for T2 = 2 T in [2^59, 3 * 2^61): a
// single-precision reciprocal root r (relative error below 2^-21.4 with the conversion's), its
// residual eps = T r^2 - 1 in integers, and the series (1 + eps)^(-1/2) = 1 - eps/2 + 3 eps^2/8 - ...,
// whose next term is below 2^-64.
TZG_HD long long inv_sqrt(long long T2) {
  // 2^44 * 2^-16 sqrt(2): r is the reciprocal root of T2's high word.
  const float r = rsqrt_seed((float)(unsigned)(T2 >> 32));
  const int r2 = float_to_int_sat(mulf(r, 17592186044416.0f * 1.41421356f));  // r 2^60
  const Limbs p = limbs(mad_wide(r2, r2, 0)), t = limbs(T2);
  long long mid = mad_wide(t.h, p.l, 1LL << 31);
  mid = mad_wide(t.l, p.h, mid);
  const long long e = mad_wide(t.h, p.h, -(1LL << 57)) + (mid >> 32);                // eps 2^57
  const int e2 = (int)(e >> 6);                                                     // eps 2^51
  const int q = high(mad_wide(e2, e2, 0));                                          // eps^2 2^70
  const Limbs d = limbs((e << 4) - ((3 * q) >> 11));                                // (eps/2 - 3/8 eps^2) 2^62
  // r (1 - d) 2^91
  return ((long long)r2 << 31) - (mad_wide(r2, d.h, 0) << 1) - (mad_wide(r2, d.l, 0) >> 31);
}

// v g / 2^61 for |v| <= 2^62, |g| <= 2^62.6 and a result up to 2^62 (a coefficient), to 2^-59 of that.
// The low half comes out odd, hence never -2^31: the halves can be negated one by one.
TZG_HD Limbs scale_coef(Limbs x, Limbs g) {
  long long mid = mad_wide(x.h, g.l, 1LL << 31);
  mid = mad_wide(x.l, g.h, mid);
  const long long s = mad_wide(x.h, g.h, 1LL << 28) + (mid >> 32);  // result / 8 + 2^28
  Limbs r;
  r.h = (int)(s >> 29);
  r.l = (int)((unsigned)s * 8u + 0x80000001u);
  return r;
}

// Rotation coefficients: c = x / N, s = y / N with N = sqrt(|x|^2 + y^2), y real; c = 1, s = 0 (to a
// rounding) for x = y = 0. G = [conj(c) s; -s c] maps (x, y) to (N, 0). Arguments: V values below 2^62.
struct RotC {
  Limbs cr, ci, s;
};
TZG_HD RotC make_rotc(long long xr, long long xi, long long y) {
  // Only for values below 2^-30 of the bound do the low words and zeros matter.
  const unsigned top = mag32(high(xr)) | mag32(high(xi)) | mag32(high(y));
  int z = clz32(top) - 2;
  if (top == 0) {
    xr += (xr | xi | y) == 0 ? 1 : 0;
    z = clz64(mag64(xr) | mag64(xi) | mag64(y) | 1ull) - 2;
  }
  const Limbs a = limbs(xr << z), b = limbs(xi << z), d = limbs(y << z);  // the largest's top bit at 2^61
  long long mid = mad_wide(a.h, a.l, 0);
  long long T = mad_wide(a.h, a.h, 0);
  mid = mad_wide(b.h, b.l, mid);
  T = mad_wide(b.h, b.h, T);
  mid = mad_wide(d.h, d.l, mid);
  T = mad_wide(d.h, d.h, T);
  const Limbs G = limbs(inv_sqrt((T << 1) + (mid >> 30)));
  RotC g;
  g.cr = scale_coef(a, G);
  g.ci = scale_coef(b, G);
  g.s = scale_coef(d, G);
  g.s.l -= y == 0 ? 1 : 0;  // exactly zero: what a step without a subdiagonal takes in must not matter
  return g;
}

// [a; b] <- [cc a + s b; conj(cc) b - s a], cc = cr + i ci; ni, ns: ci and s negated.
TZG_HD void rotate(const Starts& k, Limbs cr, Limbs ci, Limbs ni, Limbs s, Limbs ns, cfx a, cfx b, cfx& oa, cfx& ob) {
  const Limbs ax = entry_limbs(a.x), ay = entry_limbs(a.y), bx = entry_limbs(b.x), by = entry_limbs(b.y);
  oa.x = dot3(k, cr, ax, ni, ay, s, bx);
  oa.y = dot3(k, cr, ay, ci, ax, s, by);
  ob.x = dot3(k, cr, bx, ci, by, ns, ax);
  ob.y = dot3(k, cr, by, ni, bx, ns, ay);
}

TZG_HD float fx2f(long long v) {  // v as a float, from its 32-bit halves
  const Limbs a = limbs(v);
  return fmaf((float)a.h, 4294967296.0f, (float)a.l);
}

TZG_HD float abs1f(float x, float y) { return addf(fabsf(x), fabsf(y)); }

TZG_HD float exp2_int(int e) {  // 2^e, e in the normal range
  union {
    int i;
    float f;
  } u;
  u.i = (e + 127) << 23;
  return u.f;
}
TZG_HD int exponent_of(float x) {
  union {
    float f;
    int i;
  } u;
  u.f = x;
  return ((u.i >> 23) & 0xff) - 127;
}

// Wilkinson shift of the trailing 2 x 2 block [a b; y d] (y real) as a
// correction to d: d + result. The entries' differences are exact integers
// and the correction needs only its relative precision (a shift steers the
// iteration, and the correction tends to zero with y), so it is single
// precision. The same cancellation-free form as the FP64 path's. b and y are
// V values; a and d may be entries (only their difference enters).
TZG_HD cfx wilkinson_correction(cfx a, cfx b, long long y, cfx d) {
  cfx out = {0, 0};
  const float k32 = 2.3283064365386963e-10f;  // 2^-32
  const float yy = mulf(fx2f(y), k32);
  const float bcx = mulf(mulf(fx2f(b.x), k32), yy), bcy = mulf(mulf(fx2f(b.y), k32), yy);
  const float xx = mulf(fx2f(a.x - d.x), 0.5f * k32), xy = mulf(fx2f(a.y - d.y), 0.5f * k32);
  const float bc1 = abs1f(bcx, bcy), x1 = abs1f(xx, xy);
  if (bc1 < 1e-30f) return out;
  int k = exponent_of(bc1) >> 1;
  if (x1 > 0.0f) {
    const int kx = exponent_of(x1);
    if (kx > k) k = kx;
  }
  const float is = exp2_int(-k);
  const float ux = mulf(xx, is), uy = mulf(xy, is), vx = mulf(mulf(bcx, is), is), vy = mulf(mulf(bcy, is), is);
  const float zx = fmaf(ux, ux, fmaf(-uy, uy, vx)), zy = fmaf(mulf(2.0f, ux), uy, vy);
  const float u = mulf(0.5f, addf(sqrtf(fmaf(zx, zx, mulf(zy, zy))), fabsf(zx)));
  float rx = 0.0f, ry = 0.0f;
  if (u > 0.0f) {
    const float r = rsqrt_seed(u), t = mulf(u, r), h = mulf(mulf(0.5f, zy), r);
    rx = zx >= 0.0f ? t : fabsf(h);
    ry = zx >= 0.0f ? h : copysignf(t, zy);
  }
  if (fmaf(ux, rx, mulf(uy, ry)) < 0.0f) {
    rx = -rx;
    ry = -ry;
  }
  const float dx = addf(ux, rx), dy = addf(uy, ry);
  const float den = fmaf(dx, dx, mulf(dy, dy));
  if (!(den > 0.0f)) return out;
  const float f = mulf(exp2_int(k) / den, 4294967296.0f);
  // |correction| <= sqrt|bc| <= the block's norm
  out.x = -(long long)mulf(fmaf(vx, dx, mulf(vy, dy)), f);
  out.y = -(long long)mulf(fmaf(vy, dx, mulf(-vx, dy)), f);
  return out;
}

// Deflation test of the real subdiagonal y between diagonal entries d1
// (above) and d2, with the entry `up` opposite it and its neighbouring
// subdiagonals yu, yd: the Ahues-Tisseur criterion (LAPACK Working Note 122)
// at `ulps` times 2^-52, or at most kFixedSmall. All V values.
TZG_HD bool fixed_negligible(long long y, cfx d1, cfx d2, cfx up, long long yu, long long yd, int ulps = 1) {
  const long long h = y < 0 ? -y : y;
  if (h <= kFixedSmall) return true;
  unsigned long long tst = mag64(d1.x) + mag64(d1.y) + mag64(d2.x) + mag64(d2.y);
  if (tst == 0) tst = mag64(yu) + mag64(yd);
  if ((unsigned long long)h > (tst >> 52) * ulps) return false;
  const float k32 = 2.3283064365386963e-10f;
  const float h1 = mulf(fx2f(h), k32), hu = mulf(abs1f(fx2f(up.x), fx2f(up.y)), k32);
  const float ab = fmaxf(h1, hu), ba = fminf(h1, hu);
  const float dd = mulf(abs1f(fx2f(d1.x - d2.x), fx2f(d1.y - d2.y)), k32);
  const float e2 = mulf(abs1f(fx2f(d2.x), fx2f(d2.y)), k32);
  const float aa = fmaxf(e2, dd), bb = fminf(e2, dd);
  const float s = addf(aa, ab);
  const float ulp = mulf(2.220446049250313e-16f, (float)ulps);
  return mulf(ba, ab / s) <= fmaxf((float)kFixedSmall * k32, mulf(ulp, mulf(bb, aa / s)));
}

// Upper Hessenberg storage: column c holds rows 0..c+1 (0..n-1 for the last), one after another.
TZG_HD int hess_col(int c) { return c * (c + 3) / 2; }
TZG_HD int hess_idx(int r, int c) { return hess_col(c) + r; }
TZG_HD int hess_count(int n) { return n < 2 ? n : hess_col(n - 1) + n; }
// In the workspace, matrices follow one another; from n = 5 on each has an entry in front and one behind.
TZG_HD int hess_lead(int n) { return n >= 5 ? 1 : 0; }
TZG_HD int hess_stride(int n) { return hess_count(n) + 2 * hess_lead(n); }

// Entries of a unitary matrix: kFixedOne is 1 (its columns' norms stay far below the entries' bound).
constexpr int kFixedOneBits = 60;
constexpr long long kFixedOne = 1LL << kFixedOneBits;
// Where a Schur form's matrices are n^2 entries apart (n >= 5), a matrix's state is kept behind its packed form.
TZG_HD int* schur_state(cfx* packed, int n) { return (int*)(packed + n * n - 1); }

}  // namespace tzg
