// Schur forms A = Q T Q^H in 64-bit fixed point (zgeev_fixed.cuh), for ragged gradients and eigenvectors.
//
// The sweeps of zgeev_fixed_qr.cuh with every entry kept up to date: lane r of a matrix's L lanes holds the
// indices j = r, r + L, ... of T. An index inside the window [lo, hi] is a column until its rotation is known
// and a row after it; one right of the window is a column (its entries of the window's rows rotate), one above
// it is a row (its entries of the window's columns do). The same number of rows of Q, which stays in the
// workspace, rotate as rows. T is in shared memory, packed upper Hessenberg.
//
// The first shift after each deflation is the nearest unused one of a list: the forward's eigenvalues
// (gradients) or single-precision estimates (eigenvectors); then Wilkinson's.
//
// Bound by the multiplier and, with Q in the workspace, the latency of its rows, as the eigenvalue QR. Against the
// FP64 Schur forms: eigenvectors of 8,192 matrices of order 32 37.6 -> 17.4 ms, forward and gradient of
// 4,000 of orders 8 to 64 108 -> 37 ms. Orders below 5, where n^2 entries do not hold the packed form and a state,
// stay in FP64.
#pragma once

#include "zgeev_fixed_launch.cuh"

namespace tzg {

// Words of 16 bytes beside T: as qr_words, and the list of first shifts.
__host__ __device__ constexpr int schur_words(int n) { return qr_words(n) + n; }
template <int L>
inline size_t fixed_schur_shared(int n) {
  return ((size_t)(32 / L) * (qr_stride<L>(n) + schur_words(n)) + qr_slack(n)) * 16;
}

template <int L, int T>
struct SchurLane {
  Checked<cfx> H, W, Q;  // T (packed; as read and as written), Q (column-major n x n)
  int4* cur;       // as QrLane
  cfx* next;
  Checked<long long> sub;
  Starts starts;
  int rank, n, lo, m;
  cfx carry[2 * T], ld[2 * T];  // T's indices, then Q's rows
  int at[2 * T];

  // Before step 0: the entries of row lo (columns) or column lo (rows).
  __device__ __forceinline__ void begin() {
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const int j = min(rank + t * L, n - 1);
      const int first = j >= lo ? hess_idx(lo, j) : hess_idx(j, lo);
      at[t] = j >= lo ? first + 1 : hess_idx(j, lo + 1);
      carry[t] = H[first];
      ld[t] = H[at[t]];
      at[T + t] = (lo + 1) * n + j;
      carry[T + t] = Q[lo * n + j];
      ld[T + t] = Q[at[T + t]];
      if (rank + t * L == lo) *next = carry[t];
    }
  }

  __device__ __forceinline__ void sweep(int last) {
    for (int kk = 0; kk <= last; ++kk) {
      const int k = lo + kk;
      __syncwarp();
      const cfx x = *next;
      const long long y = kk < m ? sub[kk] : kZero;
      {
        const RotC g = make_rotc(x.x - kZero, x.y - kZero, y - kZero);
        if (rank == 0) {
          const int4 a = make_int4(g.cr.h, g.cr.l, g.s.h, g.s.l);
          int4* const r = cur + 2 + (kk & 3) * 2;
          cur[0] = a;
          cur[1] = make_int4(-g.ci.h, -g.ci.l, g.ci.h, g.ci.l);
          r[0] = a;
          r[1] = make_int4(g.ci.h, g.ci.l, -g.ci.h, -g.ci.l);
        }
      }
      __syncwarp();
      const int4* const row = cur + 2 + ((kk - 2) & 3) * 2;
      const int4 ra = row[0], rb = row[1];
      const bool rows = kk >= 2 && kk <= m + 1;  // rotation kk - 2 exists
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int i = rank + t * L - lo;
        const bool col = i >= kk;
        const int4* const c = col ? cur : row;
        const int4 a = c[0], b = c[1];
        cfx o, p;
        rotate(starts, Limbs{a.x, a.y}, Limbs{b.x, b.y}, Limbs{b.z, b.w}, Limbs{a.z, a.w}, Limbs{-a.z, -a.w}, carry[t],
               ld[t], o, p);
        // Columns right of the window take rotations 0 .. m - 1, indices above it rotations from step 2 on.
        const bool live = rank + t * L < n && (i >= m ? kk < m : i < 0 ? rows : kk <= m + 1);
        if (live) {
          W[at[t] - (col ? 1 : k)] = o;
          carry[t] = p;
          if (i >= m ? kk + 1 < m : kk <= m) at[t] += i > kk ? 1 : i == kk ? -1 : k + 1;
        }
        if (i == kk + 1) *next = carry[t];
        ld[t] = H[at[t]];
      }
#pragma unroll
      for (int t = 0; t < T; ++t) {
        cfx o, p;
        rotate(starts, Limbs{ra.x, ra.y}, Limbs{rb.x, rb.y}, Limbs{rb.z, rb.w}, Limbs{ra.z, ra.w},
               Limbs{-ra.z, -ra.w}, carry[T + t], ld[T + t], o, p);
        if (rows && rank + t * L < n) {
          Q[at[T + t] - n] = o;
          carry[T + t] = p;
          at[T + t] += n;
          if (kk < m) ld[T + t] = Q[at[T + t]];
        }
      }
    }
  }
};

// v 2^-e as a fixed-point value, or false if it is not finite or not below the entries' bound.
__device__ __forceinline__ bool shift_to_fixed(double v, int e, long long& out) {
  const long long bits = __double_as_longlong(v);
  const int ex = (int)((bits >> 52) & 0x7ff);
  out = 0;
  if (ex == 0) return true;
  const long long m = (bits & 0xfffffffffffffLL) | (1LL << 52);
  const int s = ex - 1075 - e;  // v 2^-e = m 2^s
  if (s > 8) return false;      // 2^61 or more (also infinities and NaN)
  if (s >= 0)
    out = m << s;
  else if (s > -54)
    out = (m + (1LL << (-s - 1))) >> -s;
  if (bits < 0) out = -out;
  return true;
}

// First shifts: eigenvalues, or single-precision estimates (n of them, or `stride` apart; null: none).
struct EigenvalueShifts {
  const double2* lam;
  const long long* offsets;  // null: n apart
  __device__ __forceinline__ bool any() const { return true; }
  __device__ __forceinline__ double2 get(long long j, int n, int k) const {
    return lam[(offsets != nullptr ? offsets[j] : j * n) + k];
  }
};
struct EstimateShifts {
  const float2* est;
  __device__ __forceinline__ bool any() const { return est != nullptr; }
  __device__ __forceinline__ double2 get(long long j, int n, int k) const {
    const float2 e = est[j * n + k];
    return make_double2(e.x, e.y);
  }
};

// What becomes of a Schur form: T's upper triangle (times a power of two) in the FP64 kernels' tiles; with `gbar`
// the gradient of the eigenvalue that position i deflated to, in vec; with `w` the eigenvalues, and the flag of a
// matrix that did not converge.
struct SchurDone {
  double2* T;
  double2* vec;
  const double2* gbar;
  const long long* offsets;  // of eigenvalues and gradients (null: n apart)
  double2* w;
  char* flag;
  __device__ __forceinline__ long long eig(long long j, int n) const { return offsets != nullptr ? offsets[j] : j * n; }
  __device__ __forceinline__ void entry(const FixedTile& t, int slot, int r, int c, double2 v) const {
    const int p = t.pos + slot, g0 = p / t.width * t.width, tw = min(t.width, t.total - g0);
    TZG_DBG_INDEX(r, t.n);
    TZG_DBG_INDEX(c, t.n);
    T[t.origin + (long long)g0 * t.n * t.n + (long long)(c * t.n + r) * tw + (p - g0)] = v;
  }
  __device__ __forceinline__ void deflated(const FixedTile& t, int slot, int i, int k) const {
    if (gbar == nullptr) return;
    const int p = t.pos + slot, g0 = p / t.width * t.width, tw = min(t.width, t.total - g0);
    vec[t.origin + (long long)g0 * t.n * t.n + (long long)i * tw + (p - g0)] = gbar[eig(t.j, t.n) + k];
  }
  __device__ __forceinline__ void eigenvalue(const FixedTile& t, int i, cfx v, int e) const {
    if (w != nullptr) w[eig(t.j, t.n) + i] = make_double2(fixed_to_double(v.x, e), fixed_to_double(v.y, e));
  }
  __device__ __forceinline__ void failed(const FixedTile& t) const {
    if (w != nullptr) flag[t.j] = (char)kNotConverged;
  }
};

// `ulps`: deflation threshold. The state (schur_state) is an exponent on entry; kStateDone on return if the
// iteration did not converge, kStateGeneral if a first shift is not below the entries' bound.
template <int L, int T, class Work, class Hint, class Done>
__global__ void __launch_bounds__(32) fixed_schur_kernel(Work work, Hint hint, Done done, cfx* __restrict__ hess,
                                                          cfx* __restrict__ q, int itmax0, int ulps, int one) {
  constexpr int TW = 32 / L;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) char fixed_smem[];
  const int lane = threadIdx.x & 31, rank = lane & (L - 1), slot = lane / L, base = lane & ~(L - 1);
  FixedTile tile;
  for (long long tix = blockIdx.x; work.tile(tix, TW, slot, tile); tix += gridDim.x) {
    const int n = tile.n, nn = n * n, count = hess_count(n), stride = qr_stride<L>(n);
    const int itmax = itmax0 > 0 ? itmax0 : default_itmax(n);
    const long long j = tile.j;
    const long long mine = tile.where + (long long)min(slot, tile.count - 1) * nn;
    int* const state = schur_state(hess + mine, n);
    const int st = slot < tile.count ? *state : kStateDone;
    bool have = st != kStateDone && st != kStateGeneral;
    if (!__any_sync(kAll, have)) continue;
    cfx* words = reinterpret_cast<cfx*>(fixed_smem);
    const Checked<cfx> sm = checked(words + 1, 0, TW * stride - 1);
    const int all = tile.count * count;
    for (int e = lane; e < all; e += 32) {
      const int t = TW == 1 ? 0 : e / count;
      sm[t * stride + (e - t * count)] = hess[tile.where + (long long)t * nn + hess_lead(n) + (e - t * count)];
    }
    cfx* const h = words + 1 + slot * stride;
    const Checked<cfx> H = checked(h, -1, count + 1 + qr_slack(n));
    words += TW * stride + slot * schur_words(n);
    SchurLane<L, T> S;
    S.H = H;
    S.W = checked(h, -1, count + 1);
    S.Q = checked(q + mine, 0, nn);
    S.cur = reinterpret_cast<int4*>(words);
    S.next = words + 10;
    S.sub = checked(reinterpret_cast<long long*>(words + 11), 0, n);
    cfx* const list = words + qr_words(n);
    S.starts = make_starts(one);
    S.rank = rank;
    S.n = n;
    if (rank == 0) H[count] = cfx{kZero, kZero};
    const bool listed = hint.any();
    if (listed) {
      bool fine = true;
      if (have)
        for (int k = rank; k < n; k += L) {
          const double2 v = hint.get(j, n, k);
          cfx f;
          fine = shift_to_fixed(v.x, st, f.x) && fine;
          fine = shift_to_fixed(v.y, st, f.y) && fine;
          const float x = mulf(fx2f(f.x), 2.3283064365386963e-10f), y = mulf(fx2f(f.y), 2.3283064365386963e-10f);
          fine = fmaf(x, x, mulf(y, y)) < 2.88e17f && fine;  // below 2^61
          list[k] = f;
        }
      const unsigned bad = __ballot_sync(kAll, !fine) >> base & (L == 32 ? kAll : (1u << (L & 31)) - 1u);
      if (bad != 0) {
        have = false;
        if (rank == 0) *state = kStateGeneral;
      }
    }
    __syncwarp();

    // The unused list entry nearest to z (distances in single precision, of exact differences); -1 without a list.
    unsigned long long used = 0;
    auto nearest = [&](cfx z) {
      float best = 3.4e38f;
      int at = 1 << 30;
      for (int k = rank; k < n; k += L) {
        if ((used >> k) & 1ull) continue;
        const float dx = mulf(fx2f(list[k].x - z.x), 2.3283064365386963e-10f);
        const float dy = mulf(fx2f(list[k].y - z.y), 2.3283064365386963e-10f);
        const float d = fmaf(dx, dx, mulf(dy, dy));
        if (d < best) {
          best = d;
          at = k;
        }
      }
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) {
        const float b = __shfl_xor_sync(kAll, best, o);
        const int a = __shfl_xor_sync(kAll, at, o);
        if (b < best || (b == best && a < at)) {
          best = b;
          at = a;
        }
      }
      return at < n ? at : 0;
    };

    int hi = have ? n - 1 : -1;
    int its = 0, kdefl = 0, status = kConverged;
    while (true) {
      int lo = 0;
      unsigned long long small = 0;
      const int top = __reduce_max_sync(kAll, hi);
      if (top < 0) break;
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int k = rank + t * L;
        bool neg = false;
        if (k >= 1 && k <= hi) {
          const long long y = H[hess_idx(k, k - 1)].x - kZero;
          const cfx d1 = H[hess_idx(k - 1, k - 1)], d2 = H[hess_idx(k, k)], up = H[hess_idx(k - 1, k)];
          const long long yu = k >= 2 ? H[hess_idx(k - 1, k - 2)].x - kZero : 0;
          const long long yd = k < hi ? H[hess_idx(k + 1, k)].x - kZero : 0;
          neg = fixed_negligible(y, cfx{d1.x - kZero, d1.y - kZero}, cfx{d2.x - kZero, d2.y - kZero},
                                 cfx{up.x - kZero, up.y - kZero}, yu, yd, ulps);
        }
        const unsigned vote = (__ballot_sync(kAll, neg) >> base) & (L == 32 ? kAll : (1u << (L & 31)) - 1u);
        small |= (unsigned long long)vote << (t * L);
      }
      // Converged positions; all groups of the warp go round together for the list's shuffles.
      bool open = hi >= 0;
      while (__any_sync(kAll, open)) {
        bool off = false;
        if (open) {
          const unsigned long long below = small & ((2ull << hi) - 1ull);
          lo = below ? 63 - clz64(below) : 0;
          off = lo == hi;
          open = off;
        }
        if (!__any_sync(kAll, off)) break;
        if (listed) {
          const cfx d = off ? H[hess_idx(hi, hi)] : cfx{kZero, kZero};
          const int k = nearest(cfx{d.x - kZero, d.y - kZero});
          if (off) {
            used |= 1ull << k;
            if (rank == 0) done.deflated(tile, slot, hi, k);
          }
        }
        if (off) {
          if (rank == 0 && hi > 0) H[hess_idx(hi, hi - 1)] = cfx{kZero, kZero};
          --hi;
          its = 0;
          kdefl = 0;
          if (hi < 0) open = false;
        }
      }
      if (hi >= 0 && its > itmax) {
        status = kNotConverged;
        hi = -1;
      }
      const int m = hi < 0 ? -2 : hi - lo + 1;
      const int steps = __reduce_max_sync(kAll, m + 2);
      if (steps == 0) continue;
      ++kdefl;
      cfx sigma = {0, 0};
      if (m > 0) {
        const cfx d = H[hess_idx(hi, hi)];
        const cfx b = H[hess_idx(hi - 1, hi)];
        const cfx e = wilkinson_correction(H[hess_idx(hi - 1, hi - 1)], cfx{b.x - kZero, b.y - kZero},
                                           H[hess_idx(hi, hi - 1)].x - kZero, d);
        sigma.x = d.x - kZero + e.x;
        sigma.y = d.y - kZero + e.y;
        if (kdefl % kExceptionalPeriod == 0) {
          const bool bottom = kdefl % (2 * kExceptionalPeriod) == 0;
          const cfx f = bottom ? d : H[hess_idx(lo, lo)];
          const long long y = H[bottom ? hess_idx(hi, hi - 1) : hess_idx(lo + 1, lo)].x - kZero;
          const long long h = mag64(y) - (mag64(y) >> 2);
          sigma.x = f.x - kZero;
          sigma.x += sigma.x < 0 ? h : -h;
          sigma.y = f.y - kZero;
        }
      }
      if (listed && __any_sync(kAll, m > 0 && its == 0)) {
        const int k = nearest(sigma);
        if (m > 0 && its == 0) sigma = list[k];
      }
      ++its;
      __syncwarp();
#pragma unroll
      for (int t = 0; t < T; ++t) {  // H - sigma I on the window
        const int i = rank + t * L - lo;
        if (i >= 0 && i < m) {
          cfx* const d = &H[hess_idx(lo + i, lo + i)];
          d->x -= sigma.x;
          d->y -= sigma.y;
          S.sub[i] = H[hess_idx(lo + i + 1, lo + i)].x;
        }
      }
      if (rank == 0) {
        S.cur[2 + 6] = make_int4(1 << 30, 0, 0, 0);  // rotation lo - 1: none
        S.cur[2 + 7] = make_int4(0, 0, 0, 0);
      }
      S.lo = m > 0 ? lo : 0;
      S.m = m;
      __syncwarp();
      S.begin();
      S.sweep(steps - 1);
      __syncwarp();
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int i = rank + t * L - lo;
        if (i >= 0 && i < m) {
          cfx* const d = &H[hess_idx(lo + i, lo + i)];
          d->x += sigma.x;
          d->y += sigma.y;
        }
      }
      if (m > 0 && rank == 0) H[hess_idx(lo, lo - 1)] = cfx{kZero, kZero};
      __syncwarp();
    }
    if (have) {
      if (status != kConverged && rank == 0) {
        *state = kStateDone;
        done.failed(tile);
      }
      for (int c = rank; c < n; c += L) {
        const cfx d = H[hess_idx(c, c)];
        done.eigenvalue(tile, c, cfx{d.x - kZero, d.y - kZero}, st);
        if (status == kConverged)
          for (int r = 0; r <= c; ++r) {
            const cfx v = H[hess_idx(r, c)];
            done.entry(tile, slot, r, c,
                       make_double2(fixed_to_double(v.x - kZero, -60), fixed_to_double(v.y - kZero, -60)));
          }
      }
    }
    __syncwarp();
  }
}

template <int L, int T, class Work, class Hint, class Done>
inline cudaError_t launch_fixed_schur(const Work& work, int n, int batch, const Hint& hint, const Done& done, cfx* hess,
                                      cfx* q, int itmax, int ulps, long long max_blocks, cudaStream_t stream) {
  constexpr int tw = 32 / L;
  const size_t bytes = fixed_schur_shared<L>(n);
  const cudaError_t err = allow_shared(fixed_schur_kernel<L, T, Work, Hint, Done>, bytes);
  if (err != cudaSuccess) return err;
  long long blocks = ((long long)batch + tw - 1) / tw;
  if (max_blocks > 0 && blocks > max_blocks) blocks = max_blocks;
  fixed_schur_kernel<L, T, Work, Hint, Done>
      <<<(unsigned)blocks, 32, bytes, stream>>>(work, hint, done, hess, q, itmax, ulps, 1);
  return cudaGetLastError();
}

// The Schur forms of the matrices of `work` (orders 5 .. n): Hessenberg forms with Q (packed at `hess`, Q at `q`,
// n^2 entries per matrix), then T to `done`.
template <class Work, class Batch>
cudaError_t launch_schur_hess(const Work& work, int n, int batch, const Batch& B, cfx* hess, cfx* q, long long max_blocks,
                              cudaStream_t stream) {
  if (n <= 8) return launch_fixed_hess<8, true>(work, n, batch, B, hess, nullptr, nullptr, max_blocks, stream, q);
  if (n <= 16) return launch_fixed_hess<16, true>(work, n, batch, B, hess, nullptr, nullptr, max_blocks, stream, q);
  if (n <= 32) return launch_fixed_hess<32, true>(work, n, batch, B, hess, nullptr, nullptr, max_blocks, stream, q);
  return launch_fixed_hess<128, true>(work, n, batch, B, hess, nullptr, nullptr, max_blocks, stream, q);
}
template <class Work, class Hint, class Done>
cudaError_t launch_schur_qr(const Work& work, int n, int batch, const Hint& hint, const Done& done, cfx* hess, cfx* q,
                            int itmax, int ulps, long long max_blocks, cudaStream_t stream) {
  if (n <= 8) return launch_fixed_schur<8, 1>(work, n, batch, hint, done, hess, q, itmax, ulps, max_blocks, stream);
  if (n <= 16) return launch_fixed_schur<8, 2>(work, n, batch, hint, done, hess, q, itmax, ulps, max_blocks, stream);
  if (n <= 32) return launch_fixed_schur<16, 2>(work, n, batch, hint, done, hess, q, itmax, ulps, max_blocks, stream);
  return launch_fixed_schur<32, 2>(work, n, batch, hint, done, hess, q, itmax, ulps, max_blocks, stream);
}

// For the FP64 kernel that finishes a matrix after launch_schur_qr: its state, read before and Q converted between
// two barriers of the warp, since the tile's regions are shared by its matrices. `packed` and `qf`: this matrix's
// slots of the two regions; Q: where its double-precision entries go (over `packed`'s region).
template <int L>
__device__ __forceinline__ int take_schur(const Group<L>& G, unsigned alive, cfx* packed, const cfx* qf, double2* Q, int n,
                                          int rs) {
  const int st = *schur_state(packed, n);
  __syncwarp(alive);
  if (st != kStateDone && st != kStateGeneral)
    for (int e = G.rank; e < n * n; e += L) {
      const cfx v = qf[e];
      Q[(long long)e * rs] = make_double2(fixed_to_double(v.x - kZero, -kFixedOneBits),
                                          fixed_to_double(v.y - kZero, -kFixedOneBits));
    }
  __syncwarp(alive);
  return st;
}

}  // namespace tzg
