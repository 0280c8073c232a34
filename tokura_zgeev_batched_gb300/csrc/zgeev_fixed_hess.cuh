// Staging and Householder reduction to upper Hessenberg form in 64-bit fixed
// point (zgeev_fixed.cuh), with real subdiagonals.
//
// A group of L lanes (a part of a warp, or a block of L = 128) holds the whole
// matrix in shared memory. The reflector of column r maps x = A(r+1.., r) to
// beta e1 with beta real: P = I - mu u u^H, u = (x - beta e1) / ||x - beta e1||,
// mu = 2 (beta - Re x0) / (beta - x0) (complex, |1 - mu| = 1), applied as P A P^H.
// Each column (then each row) is one lane's, or several lanes' when lanes are
// left over: a dot product with u (integer sums; the halves' cross terms are
// folded in every two terms, so they cannot overflow) and an update.
//
// What bounds it: the 32x32-bit multiplier, 12 instructions of four clocks a term, about 60 % busy at n = 64 by
// instruction counts and times (65,536 matrices 87 ms; the FP64 reduction 197); its shared-memory reads and writes take 75 % of that time. A
// 64 x 64 matrix is 67 KB, so an SM holds three, and L = 128 lanes each give it 12 warps. Longer unrolls (four
// terms) changed nothing.
#pragma once

#include "zgeev_fixed.cuh"
#include "zgeev_fixed_guard.cuh"
#include "zgeev_fixed_qr.cuh"

namespace tzg {

template <int L>
constexpr size_t fixed_hess_shared(int n) {
  const int tw = L >= 32 ? 1 : 32 / L;
  return (size_t)tw * fixed_stride<(L > 8 ? 8 : L)>(n * (n | 1) + n) * 16 + (L > 32 ? 32 * 8 : 0);
}

// Lane group of a warp part or a whole block.
template <int L>
struct FixedGroup {
  static constexpr int kLanes = L;
  int rank;
  unsigned mask;
  unsigned long long* scratch;  // 32 words shared by the block's warps (L > 32)
  __device__ __forceinline__ FixedGroup(unsigned long long* sc) : scratch(sc) {
    rank = threadIdx.x & (L - 1);
    const int lane = threadIdx.x & 31;
    mask = L >= 32 ? 0xffffffffu : ((1u << (L & 31)) - 1u) << (lane & ~(L - 1));
  }
  __device__ __forceinline__ void sync() const {
    if (L > 32)
      __syncthreads();
    else
      __syncwarp(mask);
  }
  // Each reduction of a block uses words of its own (`at`) and leaves a barrier behind it.
  template <class F>
  __device__ __forceinline__ unsigned long long fold(unsigned long long v, int at, F op) const {
#pragma unroll
    for (int o = (L < 32 ? L : 32) / 2; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(mask, v, o));
    if (L > 32) {
      if ((threadIdx.x & 31) == 0) scratch[at + (threadIdx.x >> 5)] = v;
      __syncthreads();
      v = scratch[at];
#pragma unroll
      for (int w = 1; w < L / 32; ++w) v = op(v, scratch[at + w]);
      __syncthreads();
    }
    return v;
  }
  __device__ __forceinline__ unsigned long long ior(unsigned long long v) const {
    return fold(v, 0, [](unsigned long long a, unsigned long long b) { return a | b; });
  }
  __device__ __forceinline__ int imax(int v) const {
    return (int)fold((unsigned long long)v, 4,
                     [](unsigned long long a, unsigned long long b) { return a > b ? a : b; });
  }
  __device__ __forceinline__ float sumf(float v) const {
    return __uint_as_float((unsigned)fold(__float_as_uint(v), 8, [](unsigned long long a, unsigned long long b) {
      return (unsigned long long)__float_as_uint(addf(__uint_as_float((unsigned)a), __uint_as_float((unsigned)b)));
    }));
  }
  __device__ __forceinline__ unsigned __int128 sum128(unsigned __int128 v) const {
#pragma unroll
    for (int o = (L < 32 ? L : 32) / 2; o > 0; o >>= 1) {
      const unsigned long long lo = __shfl_xor_sync(mask, (unsigned long long)v, o);
      const unsigned long long hi = __shfl_xor_sync(mask, (unsigned long long)(v >> 64), o);
      v += ((unsigned __int128)hi << 64) | lo;
    }
    if (L > 32) {
      if ((threadIdx.x & 31) == 0) {
        scratch[12 + 2 * (threadIdx.x >> 5)] = (unsigned long long)v;
        scratch[13 + 2 * (threadIdx.x >> 5)] = (unsigned long long)(v >> 64);
      }
      __syncthreads();
      v = 0;
#pragma unroll
      for (int w = 0; w < L / 32; ++w) v += ((unsigned __int128)scratch[13 + 2 * w] << 64) | scratch[12 + 2 * w];
      __syncthreads();
    }
    return v;
  }
};

__device__ __forceinline__ unsigned __int128 square128(long long v) {
  const unsigned long long m = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  return (unsigned __int128)m * m;
}

// |x| 2^(1023 - emax) in single precision (x's bits; exponent field at most emax), rounded down.
__device__ __forceinline__ float scaled_float(long long bits, int emax) {
  const int hi = (int)(bits >> 32), d = emax - ((hi >> 20) & 0x7ff);
  if (d > 60) return 0.0f;
  return __int_as_float(((127 - d) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)bits >> 29));
}

// round(x 2^(p + 1023 - emax)) as an entry, from the bits of x.
__device__ __forceinline__ long long to_fixed(long long bits, int emax, int p) {
  const int e = (int)((bits >> 52) & 0x7ff);
  const long long m = (bits & 0xfffffffffffffLL) | (e != 0 ? 1LL << 52 : 0LL);
  const int s = 52 - p + emax - (e != 0 ? e : 1);
  const long long v = s > 54 ? 0 : s > 0 ? (m + (1LL << (s - 1))) >> s : m << -s;
  return (bits < 0 ? -v : v) + kZero;
}

// a <- a - u mu (u^H a) on the m entries a[i * es], with u (kConj: its conjugate, and mu's) as halves in
// shared memory, the entries split among `qs` neighbouring lanes (`sub`: this lane). All lanes of a warp
// call it together; `on` says whether this lane has a vector.
struct DotPart {  // conj(u) e, one term: high products and middle products
  long long hx, hy, mx, my;
  __device__ __forceinline__ void add(Limbs ur, Limbs ui, Limbs ni, Limbs x, Limbs y, long long sx, long long sy) {
    mx = mad_wide(ur.h, x.l, sx);
    my = mad_wide(ur.h, y.l, sy);
    hx = mad_wide(ur.h, x.h, hx);
    hy = mad_wide(ur.h, y.h, hy);
    mx = mad_wide(ui.h, y.l, mx);
    my = mad_wide(ni.h, x.l, my);
    hx = mad_wide(ui.h, y.h, hx);
    hy = mad_wide(ni.h, x.h, hy);
    mx = mad_wide(ur.l, x.h, mx);
    my = mad_wide(ur.l, y.h, my);
    mx = mad_wide(ui.l, y.h, mx);
    my = mad_wide(ni.l, x.h, my);
  }
};

template <bool kConj>
__device__ __forceinline__ void reflect_fixed(const Starts& k, Checked<cfx> a, int es, int m, const int4* __restrict__ u, Limbs mur,
                                              Limbs mui, bool on, int sub, int qs) {
  DotPart w = {0, 0, 0, 0};
  long long wx = 0, wy = 0;
  if (on) {
    // Two terms between folds of the middle sums: they stay below 2^63.
    Checked<cfx> p = a + sub * es;
    const int step = qs * es;
    int i = sub;
    for (; i + qs < m; i += 2 * qs, p += 2 * step) {
      const int4 c0 = u[i], c1 = u[i + qs];
      const cfx e0 = p[0], e1 = p[step];
      const Limbs i0 = {c0.z, c0.w}, j0 = {-c0.z, -c0.w}, i1 = {c1.z, c1.w}, j1 = {-c1.z, -c1.w};
      w.add(Limbs{c0.x, c0.y}, kConj ? j0 : i0, kConj ? i0 : j0, entry_limbs(e0.x), entry_limbs(e0.y), k.half,
            k.half);
      w.add(Limbs{c1.x, c1.y}, kConj ? j1 : i1, kConj ? i1 : j1, entry_limbs(e1.x), entry_limbs(e1.y), w.mx, w.my);
      wx += w.mx >> 30;
      wy += w.my >> 30;
    }
    if (i < m) {
      const int4 c0 = u[i];
      const cfx e0 = p[0];
      const Limbs i0 = {c0.z, c0.w}, j0 = {-c0.z, -c0.w};
      w.add(Limbs{c0.x, c0.y}, kConj ? j0 : i0, kConj ? i0 : j0, entry_limbs(e0.x), entry_limbs(e0.y), k.half,
            k.half);
      wx += w.mx >> 30;
      wy += w.my >> 30;
    }
    wx += w.hx << 2;
    wy += w.hy << 2;
  }
  for (int o = 1; o < qs; o <<= 1) {
    wx += __shfl_xor_sync(0xffffffffu, wx, o);
    wy += __shfl_xor_sync(0xffffffffu, wy, o);
  }
  if (!on) return;
  // -t = -mu w; mur, mui hold mu / 2
  Limbs tx, ty;
  {
    const Limbs x = limbs(-wx), y = limbs(-wy);
    const Limbs mi = kConj ? negated(mui) : mui, ni = kConj ? mui : negated(mui);
    long long mid = mad_wide(mur.h, x.l, 1LL << 28);
    mid = mad_wide(ni.h, y.l, mid);
    mid = mad_wide(mur.l, x.h, mid);
    mid = mad_wide(ni.l, y.h, mid);
    long long hh = mad_wide(mur.h, x.h, 0);
    hh = mad_wide(ni.h, y.h, hh);
    tx = limbs((hh << 3) + (mid >> 29));
    mid = mad_wide(mur.h, y.l, 1LL << 28);
    mid = mad_wide(mi.h, x.l, mid);
    mid = mad_wide(mur.l, y.h, mid);
    mid = mad_wide(mi.l, x.h, mid);
    hh = mad_wide(mur.h, y.h, 0);
    hh = mad_wide(mi.h, x.h, hh);
    ty = limbs((hh << 3) + (mid >> 29));
  }
  Checked<cfx> p = a + sub * es;
  const int step = qs * es;
#pragma unroll 2
  for (int i = sub; i < m; i += qs, p += step) {
    const int4 c = u[i];
    const Limbs ur = {c.x, c.y}, ui = kConj ? Limbs{-c.z, -c.w} : Limbs{c.z, c.w};
    const Limbs ni = kConj ? Limbs{c.z, c.w} : Limbs{-c.z, -c.w};
    cfx e = *p;
    long long mx = mad_wide(ur.h, tx.l, k.half), my = mad_wide(ur.h, ty.l, k.half);
    long long hx = mad_wide(ur.h, tx.h, 0), hy = mad_wide(ur.h, ty.h, 0);
    mx = mad_wide(ni.h, ty.l, mx);
    my = mad_wide(ui.h, tx.l, my);
    hx = mad_wide(ni.h, ty.h, hx);
    hy = mad_wide(ui.h, tx.h, hy);
    mx = mad_wide(ur.l, tx.h, mx);
    my = mad_wide(ur.l, ty.h, my);
    mx = mad_wide(ni.l, ty.h, mx);
    my = mad_wide(ui.l, tx.h, my);
    e.x += join(hx, mx);
    e.y += join(hy, my);
    *p = e;
  }
}

// Reflector scalars of one column (the same in every lane).
struct Reflector {
  int q;            // V values are shifted left by q (right by -q) before scaling
  long long nn;     // the vector's norm, shifted alike, in [2^60, 2^61)
  Limbs gv;         // scale of u
  long long beta;   // new subdiagonal entry
  Limbs mur, mui;   // mu / 2
};

TZG_HD long long shift_by(long long v, int q) { return q >= 0 ? v << q : v >> -q; }

// The part that a real column needs too (its imaginary part does not enter here).
__device__ __forceinline__ Reflector make_real_reflector(unsigned __int128 s, long long x0r) {
  Reflector f;
  const unsigned long long shi = (unsigned long long)(s >> 64), slo = (unsigned long long)s;
  const int p = shi ? 127 - clz64(shi) : 63 - clz64(slo);
  const int sh = (p - 58) & ~1;
  const long long T = sh >= 0 ? (long long)(s >> sh) : (long long)(slo << -sh);  // [2^58, 2^60)
  f.q = 31 - sh / 2;
  {
    const Limbs t = limbs(T), g = limbs(inv_sqrt(T << 1));
    long long mid = mad_wide(t.h, g.l, 0);
    mid = mad_wide(t.l, g.h, mid);
    f.nn = (mad_wide(t.h, g.h, 0) << 4) + (mid >> 28);
  }
  const long long xr = shift_by(x0r, f.q);
  const long long a = f.nn + (xr < 0 ? -xr : xr);
  const long long beta = f.q >= 1 ? ((f.nn >> (f.q - 1)) + 1) >> 1 : f.nn << -f.q;
  f.beta = xr < 0 ? beta : -beta;
  {  // ||x - beta e1||^2 = 2 N (N + |Re x0|)
    const Limbs t = limbs(f.nn), g = limbs(a);
    long long mid = mad_wide(t.h, g.l, 0);
    mid = mad_wide(t.l, g.h, mid);
    const long long hh = mad_wide(t.h, g.h, 0);
    const bool low = hh < (1LL << 57) - 8;
    const long long g4 = inv_sqrt(low ? (hh << 4) + (mid >> 28) : (hh << 2) + (mid >> 30));
    f.gv = limbs(low ? g4 << 1 : g4);
  }
  return f;
}

__device__ __forceinline__ Reflector make_reflector(unsigned __int128 s, long long x0r, long long x0i) {
  Reflector f = make_real_reflector(s, x0r);
  const long long xr = shift_by(x0r, f.q), xi = shift_by(x0i, f.q);
  const long long a = f.nn + (xr < 0 ? -xr : xr), b = xr < 0 ? -xi : xi;
  const RotC c = make_rotc(a >> 1, 0, b >> 1);  // mu = 2 cos(phi) exp(-i phi), tan(phi) = b / a
  const long long cc = value(c.cr), ss = value(c.s);
  f.mur = limbs((long long)(((__int128)cc * cc) >> 62) | 1);
  f.mui = limbs((long long)(-(((__int128)cc * ss) >> 62)) | 1);
  return f;
}

// kQ: also forms the unitary Q of A = Q H Q^H (n x n column-major entries at q + where + slot * n^2; a row of Q is
// one lane's, as a row of A from the right), leaves every matrix that is not reduced to the FP64 kernels, and keeps
// the packed form n^2 entries apart, the state behind it (schur_state).
template <int L, bool kQ, class Work, class Batch>
__global__ void __launch_bounds__(L > 32 ? L : 32) fixed_hess_kernel(Work work, Batch B, cfx* __restrict__ hess,
                                                                     char* __restrict__ flag, int* __restrict__ state,
                                                                     cfx* __restrict__ q, int one) {
  constexpr int TW = L >= 32 ? 1 : 32 / L;
  extern __shared__ __align__(16) char fixed_smem[];
  const int slot = L >= 32 ? 0 : (threadIdx.x & 31) / L;
  FixedTile tile;
  for (long long tix = blockIdx.x; work.tile(tix, TW, slot, tile); tix += gridDim.x) {
  const int n = tile.n, ld = n | 1, nn = n * n, stride = fixed_stride<(L > 8 ? 8 : L)>(n * ld + n);
  const long long j = tile.j;
  const bool exists = slot < tile.count;
  cfx* const a = reinterpret_cast<cfx*>(fixed_smem) + slot * stride;
  const Checked<cfx> A = checked(a, 0, n * ld);
  int4* const U = reinterpret_cast<int4*>(a + n * ld);
  const FixedGroup<L> G(reinterpret_cast<unsigned long long*>(fixed_smem + (size_t)TW * stride * 16));
  const Starts k = make_starts(one);
  int st = kStateDone;  // this matrix's state; only exponents go on to the reduction
  if (exists) {
    if (!kQ && !B.valid(j)) {
      const double nan = __longlong_as_double(0x7ff8000000000000LL);
      for (int i = G.rank; i < n; i += L) put_ev(B.out(j, n) + i, make_double2(nan, nan));
      if (G.rank == 0) flag[j] = (char)kInvalidInput;
    } else {
      // Entries as they come (bits), the largest exponent, then the norm.
      const auto src = B.src(j);
      int emax = 0;
      for (int e = G.rank; e < nn; e += L) {
        const double2 z = src.load(e, n);
        emax = max(emax, max(dexp_field(z.x), dexp_field(z.y)));
        const int c = e / n;
        A[c * ld + (e - c * n)] = cfx{__double_as_longlong(z.x), __double_as_longlong(z.y)};
      }
      emax = G.imax(emax);
      if (kQ && (emax == 0x7ff || emax == 0)) {
        st = kStateGeneral;
      } else if (emax == 0x7ff || emax == 0) {  // not finite, or zero
        const double v = emax != 0 ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
        for (int i = G.rank; i < n; i += L) put_ev(B.out(j, n) + i, make_double2(v, v));
        if (G.rank == 0) flag[j] = (char)(emax != 0 ? kNonFinite : kConverged);
      } else {
        G.sync();
        st = kStateGeneral;
        float s2 = 0.0f;
        const auto size = [&](int r, int c) {
          const cfx z = A[c * ld + r];
          return max(size_of(z.x), size_of(z.y));
        };
        const bool left = left_to_fp64(G, n, emax, [&](int r, int c) {
          const cfx z = A[c * ld + r];
          const float x = scaled_float(z.x, emax), y = scaled_float(z.y, emax);
          s2 = fmaf(x, x, fmaf(y, y, s2));
          return max(size_of(z.x), size_of(z.y));
        }, size, reinterpret_cast<int*>(U));
        G.sync();
        if (!left) {
          const float top = kFixedNormMax / mulf(sqrtf(G.sumf(s2)), 1.0001f);
          const int p = exponent_of(top);
          // Fixed point. Triangular matrices are left to the FP64 kernels too (an upper triangular one's diagonal is
          // exact there).
          unsigned long long lower = 0, upper = 0;
          for (int c = G.rank; c < n; c += L)
            for (int r = 0; r < n; ++r) {
              const cfx z = A[c * ld + r];
              const cfx w = {to_fixed(z.x, emax, p), to_fixed(z.y, emax, p)};
              A[c * ld + r] = w;
              const unsigned long long v = mag64(w.x - kZero) | mag64(w.y - kZero);
              if (r > c) lower |= v;
              if (r < c) upper |= v;
            }
          if (G.ior((lower != 0 ? 1u : 0u) | (upper != 0 ? 2u : 0u)) == 3) st = emax - 1023 - p;
        }
      }
    }
    if (G.rank == 0) *(kQ ? schur_state(hess + tile.where + (long long)slot * nn, n) : state + j) = st;
  }
  const bool have = st != kStateDone && st != kStateGeneral;
  if (L > 32 ? !have : !__any_sync(0xffffffffu, have)) continue;  // block- or warp-uniform
  const Checked<cfx> Q = checked(kQ ? q + tile.where + (long long)slot * nn : q, 0, nn);
  if (kQ && have)
    for (int c = 0; c < n; ++c)
      for (int r = G.rank; r < n; r += L) Q[c * n + r] = cfx{r == c ? kFixedOne + kZero : kZero, kZero};
  G.sync();

  for (int r = 0; r + 1 < n; ++r) {
    const int m = n - r - 1;
    const Checked<cfx> x = A + r * ld + r + 1;
    unsigned __int128 s = 0;
    bool need = false;
    if (have)
      for (int i = G.rank; i < m; i += L) {
        const cfx z = {x[i].x - kZero, x[i].y - kZero};
        s += square128(z.x);
        s += square128(z.y);
        need |= i == 0 ? z.y != 0 : (z.x | z.y) != 0;
      }
    if (L > 32)
      need = __syncthreads_or(need);
    else
      need = (__ballot_sync(0xffffffffu, need) & G.mask) != 0;
    if (L > 32 ? !need : !__any_sync(0xffffffffu, need)) continue;
    s = G.sum128(s);
    Reflector f;
    if (need) {
      const long long bx = x[0].x - kZero;
      f = make_reflector(s, bx, x[0].y - kZero);
      for (int i = G.rank; i < m; i += L) {
        cfx v = x[i];
        v.x = shift_by(v.x - kZero, f.q);
        v.y = shift_by(v.y - kZero, f.q);
        if (i == 0) v.x += bx < 0 ? -f.nn : f.nn;
        const Limbs ur = scale_coef(limbs(v.x), f.gv), ui = scale_coef(limbs(v.y), f.gv);
        checked(U, 0, n)[i] = make_int4(ur.h, ur.l, ui.h, ui.l);
      }
    }
    G.sync();
    if (need && G.rank == 0) x[0] = cfx{f.beta + kZero, kZero};
    // Columns r+1 .. n-1 from the left, then all rows from the right.
    int qs = 1;
    while (2 * qs * m <= L && qs < 32) qs *= 2;
    const int per = L / qs, sub = G.rank & (qs - 1);
    for (int c0 = 0; c0 < m; c0 += per) {
      const int c = c0 + G.rank / qs;
      reflect_fixed<false>(k, A + (r + 1 + c) * ld + r + 1, 1, m, U, f.mur, f.mui, need && c < m, sub, qs);
    }
    G.sync();
    qs = 1;
    while (2 * qs * n <= L && qs < 32) qs *= 2;
    const int per2 = L / qs, sub2 = G.rank & (qs - 1);
    for (int q0 = 0; q0 < n; q0 += per2) {
      const int q = q0 + G.rank / qs;
      reflect_fixed<true>(k, A + (r + 1) * ld + q, ld, m, U, f.mur, f.mui, need && q < n, sub2, qs);
      if (kQ) reflect_fixed<true>(k, Q + (r + 1) * n + q, n, m, U, f.mur, f.mui, need && q < n, sub2, qs);
    }
    G.sync();
  }
  if (have) {
    const Checked<cfx> out =
        checked(hess + tile.where + (long long)slot * (kQ ? nn : hess_stride(n)) + hess_lead(n), 0, hess_count(n));
    for (int c = 0; c < n; ++c)
      for (int r = G.rank; r <= min(c + 1, n - 1); r += L) out[hess_idx(r, c)] = A[c * ld + r];
  }
  G.sync();
  }
}

}  // namespace tzg

