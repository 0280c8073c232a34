// Real eigenvalues in 64-bit fixed point (zgeev_fixed.cuh): staging and Householder reduction of real
// matrices; the QR iteration is the complex one (zgeev_fixed_qr.cuh), which reads the real Hessenberg form,
// takes the conjugate of each eigenvalue that deflates as its next shift, and pairs the eigenvalues at the end.
//
// Francis' double-shift iteration keeps a real matrix real at a quarter of the arithmetic, but not in fixed point: its
// shifts reach the bottom of the window through products of subdiagonal entries, which an absolute unit truncates
// (one entry at 2^-46 of the norm took 5 to 20 double sweeps per eigenvalue instead of 1.5, and 1 matrix in 10 did not
// converge), where an explicitly shifted sweep has the shift in the diagonal.
#pragma once

#include "dgeev_real.cuh"
#include "zgeev_fixed_hess.cuh"

namespace tzg {

// Words between matrices of a warp: L more than a multiple of 16, so that equal offsets use distinct banks.
template <int L>
__host__ __device__ constexpr int real_stride(int words) {
  return L >= 16 ? words : words + ((L - words) & 15);
}
template <int L>
inline size_t real_hess_shared(int n) {
  const int tw = L >= 32 ? 1 : 32 / L;
  return (size_t)(tw * real_stride<(L > 16 ? 16 : L)>(n * (n | 1) + n) + (L > 32 ? 32 : 0)) * 8;
}
// a <- a - 2 u (u . a) on the m entries a[i * es], split among `qs` neighbouring lanes; as reflect_fixed.
__device__ __forceinline__ void reflect_fixed_real(const Starts& k, Checked<long long> a, int es, int m,
                                                   const int2* __restrict__ u, bool on, int sub, int qs) {
  long long w = 0, hh = 0;
  const int step = qs * es;
  if (on) {
    Checked<long long> p = a + sub * es;
    int i = sub;
    for (; i + qs < m; i += 2 * qs, p += 2 * step) {
      const int2 c = u[i], d = u[i + qs];
      const Limbs x = entry_limbs(p[0]), y = entry_limbs(p[step]);
      long long mid = mad_wide(c.x, x.l, k.half);
      hh = mad_wide(c.x, x.h, hh);
      mid = mad_wide(d.x, y.l, mid);
      hh = mad_wide(d.x, y.h, hh);
      mid = mad_wide(c.y, x.h, mid);
      mid = mad_wide(d.y, y.h, mid);
      w += mid >> 30;
    }
    if (i < m) {
      const int2 c = u[i];
      const Limbs x = entry_limbs(p[0]);
      long long mid = mad_wide(c.x, x.l, k.half);
      hh = mad_wide(c.x, x.h, hh);
      mid = mad_wide(c.y, x.h, mid);
      w += mid >> 30;
    }
    w += hh << 2;
  }
  for (int o = 1; o < qs; o <<= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  if (!on) return;
  const Limbs t = limbs(-2 * w);
  Checked<long long> p = a + sub * es;
#pragma unroll 2
  for (int i = sub; i < m; i += qs, p += step) {
    const int2 c = u[i];
    long long mid = mad_wide(c.x, t.l, k.half);
    mid = mad_wide(c.y, t.h, mid);
    *p += join(mad_wide(c.x, t.h, 0), mid);
  }
}

// Staging and reduction, as fixed_hess_kernel with a quarter of its products. Bound by shared memory: an
// entry of an update is two 8-byte loads (one a broadcast) and a store, five of its cycles, for three products (12
// cycles of one of the SM's four multipliers).
template <int L, class T>
__global__ void __launch_bounds__(L > 32 ? L : 32) real_hess_kernel(int n, int batch, const T* __restrict__ A0,
                                                                    T* __restrict__ wr, T* __restrict__ wi,
                                                                    long long* __restrict__ work, char* __restrict__ flag,
                                                                    int one) {
  constexpr int TW = L >= 32 ? 1 : 32 / L;
  extern __shared__ __align__(16) char fixed_smem[];
  const int slot = L >= 32 ? 0 : (threadIdx.x & 31) / L;
  const int ld = n | 1, nn = n * n, stride = real_stride<(L > 16 ? 16 : L)>(n * ld + n);
  const long long j = (long long)blockIdx.x * TW + slot;
  long long* const a = reinterpret_cast<long long*>(fixed_smem) + slot * stride;
  const Checked<long long> A = checked(a, 0, n * ld);
  int2* const U = reinterpret_cast<int2*>(a + n * ld);
  const FixedGroup<L> G(reinterpret_cast<unsigned long long*>(fixed_smem) + TW * stride);
  const Starts k = make_starts(one);
  int st = kStateDone;
  if (j < batch) {
    const T* const src = A0 + j * nn;
    int emax = 0;
    for (int e = G.rank; e < nn; e += L) {
      const double z = (double)src[e];
      emax = max(emax, dexp_field(z));
      const int c = e / n;
      A[c * ld + (e - c * n)] = __double_as_longlong(z);
    }
    emax = G.imax(emax);
    if (emax == 0x7ff || emax == 0) {  // not finite, or zero
      const double v = emax != 0 ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
      for (int i = G.rank; i < n; i += L) {
        put_real(wr + j * n + i, v);
        put_real(wi + j * n + i, v);
      }
      if (G.rank == 0) flag[j] = (char)(emax != 0 ? kNonFinite : kConverged);
    } else {
      G.sync();
      st = kStateGeneral;
      float s2 = 0.0f;
      const bool left = left_to_fp64(G, n, emax, [&](int r, int c) {
        const long long z = A[c * ld + r];
        const float x = scaled_float(z, emax);
        s2 = fmaf(x, x, s2);
        return size_of(z);
      }, [&](int r, int c) { return size_of(A[c * ld + r]); }, reinterpret_cast<int*>(U));
      G.sync();
      if (!left) {
        const int p = exponent_of(kFixedNormMax / mulf(sqrtf(G.sumf(s2)), 1.0001f));
        unsigned long long lower = 0, upper = 0;  // as for complex matrices
        for (int c = G.rank; c < n; c += L)
          for (int r = 0; r < n; ++r) {
            const long long w = to_fixed(A[c * ld + r], emax, p);
            A[c * ld + r] = w;
            const unsigned long long v = mag64(w - kZero);
            if (r > c) lower |= v;
            if (r < c) upper |= v;
          }
        if (G.ior((lower != 0 ? 1u : 0u) | (upper != 0 ? 2u : 0u)) == 3) st = emax - 1023 - p;
      }
    }
    if (G.rank == 0) {
      work[(j + 1) * real_words(n) - 1] = st == kStateGeneral ? kStateDone : st;
      if (st == kStateGeneral) flag[j] = kLeftToFp64;
    }
  }
  const bool have = st != kStateDone && st != kStateGeneral;
  if (L > 32 ? !have : !__any_sync(0xffffffffu, have)) return;  // block- or warp-uniform
  G.sync();

  for (int r = 0; r + 2 < n; ++r) {
    const int m = n - r - 1;
    const Checked<long long> x = A + r * ld + r + 1;
    unsigned __int128 s = 0;
    bool need = false;
    if (have)
      for (int i = G.rank; i < m; i += L) {
        const long long z = x[i] - kZero;
        s += square128(z);
        need |= i > 0 && z != 0;
      }
    if (L > 32)
      need = __syncthreads_or(need);
    else
      need = (__ballot_sync(0xffffffffu, need) & G.mask) != 0;
    if (L > 32 ? !need : !__any_sync(0xffffffffu, need)) continue;
    s = G.sum128(s);
    long long beta = 0;
    if (need) {
      const long long b0 = x[0] - kZero;
      const Reflector f = make_real_reflector(s, b0);
      beta = f.beta;
      for (int i = G.rank; i < m; i += L) {
        long long v = shift_by(x[i] - kZero, f.q);
        if (i == 0) v += b0 < 0 ? -f.nn : f.nn;
        const Limbs c = scale_coef(limbs(v), f.gv);
        checked(U, 0, n)[i] = make_int2(c.h, c.l);
      }
    }
    G.sync();
    if (need && G.rank == 0) x[0] = beta + kZero;
    int qs = 1;
    while (2 * qs * m <= L && qs < 32) qs *= 2;
    const int per = L / qs, sub = G.rank & (qs - 1);
    for (int c0 = 0; c0 < m; c0 += per) {
      const int c = c0 + G.rank / qs;
      reflect_fixed_real(k, A + (r + 1 + c) * ld + r + 1, 1, m, U, need && c < m, sub, qs);
    }
    G.sync();
    qs = 1;
    while (2 * qs * n <= L && qs < 32) qs *= 2;
    const int per2 = L / qs, sub2 = G.rank & (qs - 1);
    for (int q0 = 0; q0 < n; q0 += per2) {
      const int q = q0 + G.rank / qs;
      reflect_fixed_real(k, A + (r + 1) * ld + q, ld, m, U, need && q < n, sub2, qs);
    }
    G.sync();
  }
  if (have) {
    const Checked<long long> out = checked(work + j * real_words(n), 0, hess_count(n));
    for (int c = 0; c < n; ++c)
      for (int r = G.rank; r <= min(c + 1, n - 1); r += L) out[hess_idx(r, c)] = A[c * ld + r];
  }
}

}  // namespace tzg
