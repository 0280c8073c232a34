// Eigenvalues of upper Hessenberg matrices in 64-bit fixed point (zgeev_fixed.cuh).
//
// A group of L lanes of a warp owns a matrix, which stays in shared memory
// (packed upper Hessenberg, real subdiagonals) from the first sweep to the
// last. A sweep is one explicitly shifted QR step on the active window
// [lo, hi], H - sigma I = Q R, H' = R Q + sigma I, with rotations
// [conj(c) s; -s c], s real, so that subdiagonals stay real. Lane r holds the
// indices j = lo + r, lo + r + L, ...: until rotation j is known index j is
// column j, which receives rotation k of the rows (k, k+1) in step k and
// carries its entry of row k+1 in registers; from step j + 1 on it is row j,
// which receives rotation k-2 of the columns (k-2, k-1) in step k and carries
// its entry of column k-1. So every index of the window does one complex
// rotation in each of the window's steps, whether it is still a column or
// already a row, each entry is loaded and stored once per half sweep, and the
// only chain is rotation -> next column's entry -> next rotation. After the
// window's last row, rotation hi is the phase that makes R(hi, hi) real.
//
// Matrices of one warp run their sweeps in lockstep; a matrix that is done, or whose
// window is shorter, has its lanes idle until the others' step count is reached.
#pragma once

#include "zgeev_fixed.cuh"
#include "zgeev_internal.h"
#include "zgeev_lane.cuh"

namespace tzg {

// Per-matrix state between the kernels: a power-of-two exponent, or one of these.
constexpr int kStateGeneral = -2147483647;  // left to the FP64 kernels (kStateDone: nothing left to do)

// Entries of 16 bytes between consecutive matrices of a warp in shared memory: lanes of a quarter
// warp reading consecutive entries of their own matrices then use different banks.
template <int L>
__host__ __device__ constexpr int fixed_stride(int count) {
  return L >= 8 ? count : (count + 7 - ((count + 7 - L) & 7));
}
// Words of 16 bytes that a matrix uses beside its entries: the current rotation as columns take it ({c.re, s},
// {-c.im, c.im}), the last four as rows do ({c.re, s}, {c.im, -c.im}), the next column's entry, and the
// subdiagonals of the sweep's start.
__host__ __device__ constexpr int qr_words(int n) { return 2 + 8 + 1 + (n + 1) / 2; }
// A matrix has one entry in front (row lo of column lo - 1 for lo = 0) and one behind (row n of
// column n - 1) its packed form; lanes without work in a step may read, not write, up to qr_slack
// entries further.
__host__ __device__ constexpr int qr_slack(int n) { return n + 8; }
template <int L>
__host__ __device__ constexpr int qr_stride(int n) {
  return fixed_stride<L>(hess_count(n) + 2);
}

// kGlobal: the matrices stay in the workspace (in cache) instead of shared memory.
template <int L, bool kGlobal>
inline size_t fixed_qr_shared(int n) {
  return ((size_t)(32 / L) * ((kGlobal ? 0 : qr_stride<L>(n)) + qr_words(n)) + (kGlobal ? 0 : qr_slack(n))) * 16;
}

// w 2^e rounded to nearest, with integer instructions unless the result is outside the normal range.
__device__ __forceinline__ double fixed_to_double(long long w, int e) {
  const unsigned long long m = w < 0 ? 0ull - (unsigned long long)w : (unsigned long long)w;
  if (m == 0) return 0.0;
  const int z = clz64(m), ex = e + 63 - z + 1023;
  const unsigned long long sign = w < 0 ? 1ull << 63 : 0ull;
  if (ex < 1 || ex > 2045) {
    const int f = e + 62, a = f / 2, b = f - a;
    return (double)w * 2.168404344971009e-19 * pow2(a) * pow2(b);  // 2^-62
  }
  const unsigned long long r = ((m << z) >> 10) + 1 >> 1;  // 2^52 .. 2^53
  return __longlong_as_double((long long)(sign | (((unsigned long long)(ex - 1) << 52) + r)));
}

// Batches of real matrices (n >= 3). Their workspace, n^2 words of 8 bytes for each, holds for each its packed real
// Hessenberg form and a word with its state, one after another, and behind these `scratch`: room for the complex
// iterates of some of them at a time. Eigenvalues go to wr and wi; flag is kLeftToFp64 for a matrix that the
// FP64 kernel solves.
constexpr char kLeftToFp64 = 100;
struct RealBatch {
  const long long* packed;
  void* wr;
  void* wi;
  bool single;
  cfx* scratch;
  long long room;  // of scratch, in entries
  __device__ __forceinline__ void put(long long i, double re, double im) const {
    if (single) {
      static_cast<float*>(wr)[i] = (float)re;
      static_cast<float*>(wi)[i] = (float)im;
    } else {
      static_cast<double*>(wr)[i] = re;
      static_cast<double*>(wi)[i] = im;
    }
  }
};
template <class Batch>
constexpr bool kRealBatch = false;
template <>
constexpr bool kRealBatch<RealBatch> = true;
TZG_HD int real_words(int n) { return hess_count(n) + 1; }
// Eigenvalues of a real matrix are conjugates of each other, or real, if they are so to this many units (2^-30 of the
// norm). Where that leaves a choice (two of them closer than this), or finds no partner, the FP64 kernel, whose
// iteration keeps conjugates, solves the matrix.
constexpr long long kConjugateUnits = 1LL << 31;
__device__ __forceinline__ bool conjugates(cfx a, cfx b) {
  return mag64(a.x - b.x) <= (unsigned long long)kConjugateUnits &&
         mag64(a.y - kZero + (b.y - kZero)) <= (unsigned long long)kConjugateUnits;
}
// Two eigenvalues so close that their conjugates, if found where they must be, will have two partners each.
__device__ __forceinline__ bool together(cfx a, cfx b) {
  return mag64(a.x - b.x) <= (unsigned long long)(kConjugateUnits / 4) &&
         mag64(a.y - b.y) <= (unsigned long long)(kConjugateUnits / 4);
}
__device__ __forceinline__ bool nearly_real(cfx a) {
  return mag64(a.y - kZero) <= (unsigned long long)(kConjugateUnits / 2);
}

// Everything a lane keeps during a sweep. What bounds it: the 32x32-bit multiplier, one warp
// instruction in four clocks of a sub-partition (a rotation is 36 of them, its coefficients 22), about 60 % busy
// by instruction counts and times (16,384 matrices of n = 64 in the workspace, 24 warps per SM; the counters give the
// pipe's instructions, 41 % of its peak, not how long a product holds it); the rest is the chain of a step. Making rotation k + 1 beside step
// k's work (18 more multiplications and two more loads in every lane) was slower: 16,384 matrices of n = 64 87.2 -> 116.5
// ms, 10,000 of n = 32 7.9 -> 9.0.
template <int L, int T>
struct QrLane {
  Checked<cfx> H;  // packed matrix as read (lanes without work read beyond it)
  Checked<cfx> W;  // as written
  int4* cur;       // current rotation for columns; then the ring of rows' rotations
  cfx* next;       // entry (k, k) that rotation k is made from (L > 1)
  Checked<long long> sub;  // subdiagonals of the window
  Starts starts;
  int rank, lo, m;
  cfx carry[T];  // this lane's entries in flight, one per index
  cfx ld[T];     // entries that the next step takes in
  int at[T];     // and where they come from

  // The steps of one sweep, `U` indices per lane in use.
  template <int U>
  __device__ __forceinline__ void sweep(int last) {
    for (int kk = 0; kk <= last; ++kk) {
      const int k = lo + kk;
      __syncwarp();
      cfx x = carry[0];
      if (L > 1) {
        x = *next;
      } else {
#pragma unroll
        for (int t = 1; t < U; ++t)
          if (kk == t) x = carry[t];
      }
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
      int4 ca[U], cb[U];
#pragma unroll
      for (int t = 0; t < U; ++t) {
        const int4* const c = rank + t * L >= kk ? cur : row;
        ca[t] = c[0];
        cb[t] = c[1];
      }
      cfx o[U];
#pragma unroll
      for (int t = 0; t < U; ++t) {
        const int4 a = ca[t], b = cb[t];
        rotate(starts, Limbs{a.x, a.y}, Limbs{b.x, b.y}, Limbs{b.z, b.w}, Limbs{a.z, a.w}, Limbs{-a.z, -a.w}, carry[t],
               ld[t], o[t], carry[t]);
      }
      const bool on = kk <= m + 1;
#pragma unroll
      for (int t = 0; t < U; ++t) {
        const int i = rank + t * L;
        if (on && i < m) W[at[t] - (i >= kk ? 1 : k)] = o[t];
        if (kk <= m) at[t] += i > kk ? 1 : i == kk ? -1 : k + 1;
        if (L > 1 && i == kk + 1) *next = carry[t];
        ld[t] = H[at[t]];
      }
    }
  }

  __device__ __forceinline__ void run(int last, int used) {
    if constexpr (T == 1) {
      sweep<1>(last);
    } else if constexpr (T == 2) {
      if (used <= 1)
        sweep<1>(last);
      else
        sweep<2>(last);
    } else {
      static_assert(T == 4, "indices per lane");
      if (used <= 1)
        sweep<1>(last);
      else if (used == 2)
        sweep<2>(last);
      else if (used == 3)
        sweep<3>(last);
      else
        sweep<4>(last);
    }
  }
};

// Some matrices of one order that a warp (or block) takes together.
struct FixedTile {
  int n, count;     // order, matrices (the slots 0 .. count - 1)
  long long j;      // this slot's matrix
  long long where;  // first entry of slot 0's packed form in the workspace (slots follow one another)
  // Of the run of matrices of this order: its first entry where they are n^2 apart, its length, slot 0's position
  // in it, and the matrices that a warp of the FP64 kernels takes together.
  long long origin;
  int total, pos, width;
};

// Work of a uniform batch: matrices 0 .. batch - 1 in order, `tw` to a tile.
// `square`: n^2 entries apart in the workspace.
struct UniformWork {
  int n, batch;
  bool square = false;
  int width = 32;
  __device__ __forceinline__ bool tile(long long t, int tw, int slot, FixedTile& out) const {
    const long long j0 = t * tw;
    if (j0 >= batch) return false;
    out.n = n;
    out.count = (int)min((long long)tw, batch - j0);
    out.j = j0 + slot;
    out.where = j0 * (square ? n * n : hess_stride(n));
    out.origin = 0;
    out.total = batch;
    out.pos = (int)j0;
    out.width = width;
    return true;
  }
};

// `itmax` 0: the default for each order.
template <int L, int T, bool kGlobal, class Work, class Batch>
__global__ void __launch_bounds__(32) fixed_qr_kernel(Work work, Batch B, cfx* __restrict__ hess,
                                                       char* __restrict__ flag, int itmax0, int* __restrict__ state,
                                                       int one) {
  constexpr int TW = 32 / L;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) char fixed_smem[];
  const int lane = threadIdx.x & 31, rank = lane & (L - 1), slot = lane / L, base = lane & ~(L - 1);
  // A block takes every gridDim-th tile.
  FixedTile tile;
  for (long long tix = blockIdx.x; work.tile(tix, TW, slot, tile); tix += gridDim.x) {
  const int n = tile.n, count = hess_count(n), stride = qr_stride<L>(n);
  const int itmax = itmax0 > 0 ? itmax0 : default_itmax(n);
  const long long j = tile.j;
  // Whole warps stay together; lanes without a matrix keep an empty window.
  constexpr bool kReal = kRealBatch<Batch>;
  int st = kStateDone;
  if (slot < tile.count) {
    if constexpr (kReal)
      st = (int)B.packed[(j + 1) * real_words(n) - 1];
    else
      st = state[j];
  }
  const bool have = st != kStateDone && st != kStateGeneral;
  if (!__any_sync(kAll, have)) continue;
  cfx* h;
  cfx* words = reinterpret_cast<cfx*>(fixed_smem);
  if constexpr (kReal) {
    if (kGlobal) {
      h = B.scratch + ((long long)blockIdx.x * TW + slot) * (count + 2) + 1;
    } else {
      h = words + 1 + slot * stride;
      words += TW * stride;
    }
    if (have) {
      const long long* const src = B.packed + j * real_words(n);
      for (int e = rank; e < count; e += L) checked(h, 0, count)[e] = cfx{src[e], kZero};
    }
    __syncwarp();
  } else if (kGlobal) {
    h = hess + tile.where + (long long)min(slot, tile.count - 1) * hess_stride(n) + 1;
  } else {
    const Checked<cfx> sm = checked(words + 1, 0, TW * stride - 1);
    const int all = tile.count * count;
    for (int e = lane; e < all; e += 32) {
      const int t = TW == 1 ? 0 : e / count;
      sm[t * stride + (e - t * count)] = hess[tile.where + t * hess_stride(n) + hess_lead(n) + (e - t * count)];
    }
    h = words + 1 + slot * stride;
    words += TW * stride;
  }
  words += slot * qr_words(n);
  const Checked<cfx> H = checked(h, -1, count + 1 + qr_slack(n));
  QrLane<L, T> Q;
  Q.H = H;
  Q.W = checked(h, -1, count + 1);
  Q.cur = reinterpret_cast<int4*>(words);
  Q.next = words + 10;
  Q.sub = checked(reinterpret_cast<long long*>(words + 11), 0, n);
  Q.starts = make_starts(one);
  Q.rank = rank;
  if (rank == 0) H[count] = cfx{kZero, kZero};  // row n of the last column
  __syncwarp();

  int hi = have ? n - 1 : -1;
  int its = 0, kdefl = 0, status = kConverged;
  bool follow = false;  // a real matrix's next shift is the conjugate of the eigenvalue below the window
#ifdef TOKURA_DEBUG_BOUNDS
  int sweeps = 0;
#endif
  while (true) {
    // Deflation: one scan of the subdiagonals gives the window.
    int lo = 0;
    unsigned long long small = 0;
    const int top = __reduce_max_sync(kAll, hi);
    if (top < 0) break;
#pragma unroll
    for (int t = 0; t < T; ++t) {
      if (t * L > top) break;
      const int k = rank + t * L;
      bool neg = false;
      if (k >= 1 && k <= hi) {
        const long long y = H[hess_idx(k, k - 1)].x - kZero;
        const cfx d1 = H[hess_idx(k - 1, k - 1)], d2 = H[hess_idx(k, k)], up = H[hess_idx(k - 1, k)];
        const long long yu = k >= 2 ? H[hess_idx(k - 1, k - 2)].x - kZero : 0;
        const long long yd = k < hi ? H[hess_idx(k + 1, k)].x - kZero : 0;
        neg = fixed_negligible(y, cfx{d1.x - kZero, d1.y - kZero}, cfx{d2.x - kZero, d2.y - kZero},
                               cfx{up.x - kZero, up.y - kZero}, yu, yd);
      }
      if (L == 1) {
        small |= (unsigned long long)neg << k;
      } else {
        const unsigned vote = (__ballot_sync(kAll, neg) >> base) & (L == 32 ? kAll : (1u << (L & 31)) - 1u);
        small |= (unsigned long long)vote << (t * L);
      }
    }
    const int last = hi;
    while (hi >= 0) {
      const unsigned long long below = small & ((2ull << hi) - 1ull);
      lo = below ? 63 - clz64(below) : 0;
      if (lo < hi) break;
      if (kReal) {
        const cfx d = H[hess_idx(hi, hi)];
        follow = !nearly_real(d) && !(follow && conjugates(d, H[hess_idx(hi + 1, hi + 1)]));
      }
      // Converged: row hi becomes the (zero) row under the next window.
      if (rank == 0) H[hess_idx(hi, hi - 1)] = cfx{kZero, kZero};
      --hi;
      its = 0;
      kdefl = 0;
    }
    if constexpr (kReal && L * T > 32) {
      // Two eigenvalues at one place (or a real one with a partner) will not pair: no need to see the others. From order
      // 33 on (16,384 of order 64: projections 63.5 -> 54.4 ms, permutations 134 -> 112, Gaussian ones 61.2 -> 60.4); below,
      // Gaussian ones pay for it (10,000 of 32 5.77 -> 5.84, 65,536 of 16 5.39 -> 5.87, 300,000 of 4 0.98 -> 1.10).
      if (__any_sync(kAll, hi < last)) {
        bool clash = false;
        for (int p = last; p > hi; --p) {
          const cfx d = H[hess_idx(p, p)];
          const bool real = nearly_real(d);
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const int i = rank + t * L;
            if (i <= p || i >= n) continue;
            const cfx e = H[hess_idx(i, i)];
            clash |= together(d, e) || (real && conjugates(d, e));
          }
        }
        const unsigned vote = __ballot_sync(kAll, clash) >> base;
        if ((L == 32 ? vote : vote & ((1u << (L & 31)) - 1u)) != 0) {
          status = kNotConverged;
          hi = -1;
        }
      }
    }
    if (hi >= 0 && its > itmax) {
      status = kNotConverged;
      hi = -1;
    }
    const int m = hi < 0 ? -2 : hi - lo + 1;
    const int steps = __reduce_max_sync(kAll, m + 2);
    if (steps == 0) continue;
    ++its;
    ++kdefl;
#ifdef TOKURA_DEBUG_BOUNDS
    if (m > 0) ++sweeps;
#endif
    cfx sigma = {0, 0};
    if (m > 0) {
      const cfx d = H[hess_idx(hi, hi)];
      if (kdefl % kExceptionalPeriod == 0) {  // ad hoc, towards zero: no larger than the matrix's norm
        const bool bottom = kdefl % (2 * kExceptionalPeriod) == 0;
        const cfx f = bottom ? d : H[hess_idx(lo, lo)];
        const long long y = H[bottom ? hess_idx(hi, hi - 1) : hess_idx(lo + 1, lo)].x - kZero;
        const long long h = mag64(y) - (mag64(y) >> 2);
        sigma.x = f.x - kZero;
        sigma.x += sigma.x < 0 ? h : -h;
        sigma.y = f.y - kZero;
      } else if (kReal && follow && its == 1) {
        const cfx e = H[hess_idx(hi + 1, hi + 1)];
        sigma.x = e.x - kZero;
        sigma.y = kZero - e.y;
      } else {
        const cfx b = H[hess_idx(hi - 1, hi)];
        const cfx e = wilkinson_correction(H[hess_idx(hi - 1, hi - 1)], cfx{b.x - kZero, b.y - kZero},
                                           H[hess_idx(hi, hi - 1)].x - kZero, d);
        sigma.x = d.x - kZero + e.x;
        sigma.y = d.y - kZero + e.y;
      }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < T; ++t) {  // H - sigma I
      const int jj = min(lo + rank + t * L, n - 1);
      if (rank + t * L < m) {
        cfx* const d = &H[hess_idx(jj, jj)];
        d->x -= sigma.x;
        d->y -= sigma.y;
      }
      Q.at[t] = hess_idx(lo, jj) + 1;
      Q.carry[t] = H[hess_idx(lo, jj)];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const int i = rank + t * L, jj = lo + i;
      Q.ld[t] = H[Q.at[t]];
      if (i < m) Q.sub[i] = H[hess_idx(jj + 1, jj)].x;
    }
    if (rank == 0) {
      *Q.next = Q.carry[0];
      Q.cur[2 + 6] = make_int4(1 << 30, 0, 0, 0);  // rotation lo - 1: none
      Q.cur[2 + 7] = make_int4(0, 0, 0, 0);
    }
    Q.lo = lo;
    Q.m = m;
    const int used = (steps - 2 + L - 1) / L;
    Q.run(steps - 1, used);
    __syncwarp();
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const int jj = lo + rank + t * L;
      if (rank + t * L < m) {
        cfx* const d = &H[hess_idx(jj, jj)];
        d->x += sigma.x;
        d->y += sigma.y;
      }
    }
    // Row lo's index also wrote beside the window; a split stays one whatever becomes of its neighbours.
    if (m > 0 && rank == 0) H[hess_idx(lo, lo - 1)] = cfx{kZero, kZero};
    __syncwarp();
  }
  if constexpr (kReal) {
    // Pairs, in the order of their first members. Anything unclear is left to the FP64 kernel.
    unsigned long long reals = 0, leads = 0;
    bool clear = status == kConverged;
    int partner[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const int i = rank + t * L;
      int found = 0;
      partner[t] = i;
      if (have && i < n) {
        const cfx d = H[hess_idx(i, i)];
        for (int c = 0; c < n; ++c)
          if (c != i && conjugates(d, H[hess_idx(c, c)])) {
            ++found;
            partner[t] = c;
          }
        clear = clear && found == (nearly_real(d) ? 0 : 1);
      }
      const bool one = have && i < n && found == 0, lead = have && i < n && partner[t] > i;
      if (L == 1) {
        reals |= (unsigned long long)one << i;
        leads |= (unsigned long long)lead << i;
      } else {
        const unsigned part = L == 32 ? kAll : (1u << (L & 31)) - 1u;
        reals |= (unsigned long long)((__ballot_sync(kAll, one) >> base) & part) << (t * L);
        leads |= (unsigned long long)((__ballot_sync(kAll, lead) >> base) & part) << (t * L);
      }
    }
    const unsigned unclear = __ballot_sync(kAll, !clear) >> base;
    clear = (L == 32 ? unclear : unclear & ((1u << (L & 31)) - 1u)) == 0;
    if (have && clear) {
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int i = rank + t * L, p = partner[t];
        if (i >= n || p < i) continue;
        const unsigned long long before = (1ull << i) - 1ull;
        const long long at = j * n + __popcll(reals & before) + 2 * __popcll(leads & before);
        const cfx d = H[hess_idx(i, i)], e = H[hess_idx(p, p)];
        if (p == i) {
          B.put(at, fixed_to_double(d.x - kZero, st), 0.0);
        } else {
          const double re = fixed_to_double(d.x - kZero + (e.x - kZero), st - 1);
          const double im = fabs(fixed_to_double(d.y - e.y, st - 1));
          B.put(at, re, im);
          B.put(at + 1, re, -im);
        }
      }
    }
    if (have && rank == 0) flag[j] = clear ? (char)kConverged : kLeftToFp64;
  } else if (have) {
    for (int i = rank; i < n; i += L) {
      const cfx d = H[hess_idx(i, i)];
      put_ev(B.out(j, n) + i, make_double2(fixed_to_double(d.x - kZero, st), fixed_to_double(d.y - kZero, st)));
    }
    if (rank == 0) flag[j] = (char)status;
  }
#ifdef TOKURA_DEBUG_BOUNDS
  if (have && rank == 0) dbg_record_sweeps(j, sweeps);
#endif
  __syncwarp();
  }
}

}  // namespace tzg
