// Launches of the fixed-point eigenvalue kernels (zgeev_fixed_hess.cuh, zgeev_fixed_qr.cuh).
#pragma once

#include "zgeev_fixed_hess.cuh"
#include "zgeev_fixed_qr.cuh"

namespace tzg {

// Shared memory above the default limit is granted per kernel, for all threads of the process: always as much as the
// largest launch of any kernel here takes (the reduction's at order 64), so that no call lowers what another has been
// granted and is about to use.
template <class Kernel>
inline cudaError_t allow_shared(Kernel kernel, size_t bytes) {
  constexpr size_t kDefault = 48 * 1024, kMost = fixed_hess_shared<128>(kMaxN);
  if (bytes <= kDefault) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost);
}

// Staging and Hessenberg reduction of the matrices of `work`, of order n at most and `batch` of them at
// most, in at most `max_blocks` blocks (0: no limit); a block takes several tiles then.
template <int L, bool kQ = false, class Work, class Batch>
inline cudaError_t launch_fixed_hess(const Work& work, int n, int batch, const Batch& B, cfx* hess, char* flag,
                                     int* state, long long max_blocks, cudaStream_t stream, cfx* q = nullptr) {
  constexpr int tw = L >= 32 ? 1 : 32 / L;
  const size_t bytes = fixed_hess_shared<L>(n);
  const cudaError_t err = allow_shared(fixed_hess_kernel<L, kQ, Work, Batch>, bytes);
  if (err != cudaSuccess) return err;
  long long blocks = ((long long)batch + tw - 1) / tw;
  if (max_blocks > 0 && blocks > max_blocks) blocks = max_blocks;
  fixed_hess_kernel<L, kQ, Work, Batch>
      <<<(unsigned)blocks, L > 32 ? L : 32, bytes, stream>>>(work, B, hess, flag, state, q, 1);
  return cudaGetLastError();
}

// The QR likewise.
template <int L, int T, bool kGlobal, class Work, class Batch>
inline cudaError_t launch_fixed_qr(const Work& work, int n, int batch, const Batch& B, cfx* hess, char* flag, int itmax,
                                   int* state, long long max_blocks, cudaStream_t stream) {
  constexpr int tw = 32 / L;
  const size_t bytes = fixed_qr_shared<L, kGlobal>(n);
  const cudaError_t err = allow_shared(fixed_qr_kernel<L, T, kGlobal, Work, Batch>, bytes);
  if (err != cudaSuccess) return err;
  long long blocks = ((long long)batch + tw - 1) / tw;
  if (max_blocks > 0 && blocks > max_blocks) blocks = max_blocks;
  fixed_qr_kernel<L, T, kGlobal, Work, Batch>
      <<<(unsigned)blocks, 32, bytes, stream>>>(work, B, hess, flag, itmax, state, 1);
  return cudaGetLastError();
}

// Eigenvalues in fixed point (zgeev_fixed.cuh); matrices it leaves keep kStateGeneral in `state`.
// Lanes per matrix: few for batches that fill the GPU, more for small ones. Measured (whole call, ms):
//   n = 4:  1,048,576 matrices 2.9 / 3.2 / 4.1 at 1 / 2 / 4 lanes, 16 matrices 0.092 / 0.076 / 0.064;
//   n = 8:  262,144 matrices 5.2 / 4.4 / 4.5 / 5.9 at 1 / 2 / 4 / 8, 4,000 0.46 / 0.30 / 0.22 / 0.20;
//   n = 16: 65,536 matrices 6.7 / 6.9 / 8.9 at 4 / 8 / 16, 4,000 0.76 / 0.69 / 0.79, 300 0.69 / 0.51 / 0.41;
//   n = 24: 30,000 matrices 10.0 / 11.7 / 16.0 at 8 / 16 / 32 (16 lanes leave 8 of 32 places empty);
//   n = 32: 10,000 matrices 9.0 / 8.0 / 9.8 at 8 / 16 / 32, 1,000 2.1 / 1.6 / 1.5.
// Above n = 32 shared memory holds few matrices (6 per SM at n = 64), so batches of more than those
// stay in the workspace, which the caches hold: n = 64, 8,192 matrices 57.7 ms in shared memory, 46 ms so
// (304 matrices: 4.9 against 6.1 ms). 32 lanes run best in 24 warps per SM (16,384 of n = 64: 92.0 / 88.0 / 87.2 / 97.9 ms
// at 16 / 20 / 24 / 32), 16 lanes in as many as 128 registers or, from about 85 MB, the L2 cache allow: 12 / 14 / 16 warps
// 39.0 / 38.5 / 35.6 (30,000 of n = 36), 37.8 / 36.8 / 36.4 (20,000 of 42), 53.3 / 52.2 / 52.8 (20,000 of 48; 32 lanes 55.7),
// 94.4 / 93.0 / 95.5 (16,384 of 64).
// Real matrices leave scratch for the complex iterates of 4 in 9 of them, used from 1.7 times the matrices that shared
// memory holds: n = 64, 3,000 matrices 18.7 ms so (1,300 blocks) and 17.1 in shared memory (912), 6,000 25.8 and 30.8,
// 16,384 62.0 and 81.9. At 16 lanes they need 32 matrices per SM to gain: n = 42, 9,000 matrices 14.0 and 13.8, 15,000 20.5
// and 22.9, 30,000 37.8 and 45.3; n = 48, 15,000 28.5 and 30.2.
template <class Batch>
cudaError_t launch_fixed_shape(const UniformWork& work, int n, int batch, int sms, const Batch& B, cfx* hess,
                               char* flag, int itmax, int* state, cudaStream_t stream) {
  // Whether a batch is small enough for `lanes` lanes per matrix and `warps` warps per SM.
  auto fits = [&](int lanes, int warps) { return (long long)batch * lanes <= (long long)sms * 32 * warps; };
#define TZG_FIXED_QR(L, T, G, BLOCKS) \
  return launch_fixed_qr<L, T, G>(work, n, batch, B, hess, flag, itmax, state, BLOCKS, stream)
  if (n <= 4) {
    if (fits(4, 8)) TZG_FIXED_QR(4, 1, false, 0);
    if (fits(2, 16)) TZG_FIXED_QR(2, 2, false, 0);
    TZG_FIXED_QR(1, 4, false, 0);
  }
  if (n <= 8) {
    if (fits(8, 8)) TZG_FIXED_QR(8, 1, false, 0);
    if (fits(4, 16)) TZG_FIXED_QR(4, 2, false, 0);
    TZG_FIXED_QR(2, 4, false, 0);
  }
  if (n <= 16) {
    if (fits(16, 8)) TZG_FIXED_QR(16, 1, false, 0);
    if (fits(8, 16)) TZG_FIXED_QR(8, 2, false, 0);
    TZG_FIXED_QR(4, 4, false, 0);
  }
  if (n <= 32) {
    if (fits(32, 8)) TZG_FIXED_QR(32, 1, false, 0);
    if (n > 24 || fits(16, 16)) TZG_FIXED_QR(16, 2, false, 0);
    TZG_FIXED_QR(8, 4, false, 0);
  }
  // Matrices that shared memory holds on all SMs (228 KB each, 1 KB of it reserved per block).
  const long long resident = (long long)sms * (233472 / (fixed_qr_shared<32, false>(n) + 1024));
  const int warps16 = n <= 42 ? 16 : 14;  // per SM, at 16 lanes
  if constexpr (kRealBatch<Batch>) {
    const long long places = (B.room - qr_slack(n)) / (hess_count(n) + 2);
    if (n <= 48 && places >= sms * 32LL) TZG_FIXED_QR(16, 4, true, sms * warps16);
    const long long blocks = min((long long)sms * 24, places);
    if (10 * blocks < 17 * resident) TZG_FIXED_QR(32, 2, false, 0);
    TZG_FIXED_QR(32, 2, true, blocks);
  } else {
    if (batch <= resident) TZG_FIXED_QR(32, 2, false, 0);
    if (n <= 48 && !fits(16, 12)) TZG_FIXED_QR(16, 4, true, sms * warps16);
    TZG_FIXED_QR(32, 2, true, sms * 24);
  }
#undef TZG_FIXED_QR
}

template <class Batch>
cudaError_t launch_fixed(int n, int batch, int sms, const Batch& B, cfx* hess, char* flag, int itmax, int* state,
                         cudaStream_t stream) {
  cudaError_t err;
  const UniformWork work{n, batch};
  if (n <= 4)
    err = launch_fixed_hess<4>(work, n, batch, B, hess, flag, state, 0, stream);
  else if (n <= 8)
    err = launch_fixed_hess<8>(work, n, batch, B, hess, flag, state, 0, stream);
  else if (n <= 16)
    err = launch_fixed_hess<16>(work, n, batch, B, hess, flag, state, 0, stream);
  else if (n <= 32)
    err = launch_fixed_hess<32>(work, n, batch, B, hess, flag, state, 0, stream);
  else
    err = launch_fixed_hess<128>(work, n, batch, B, hess, flag, state, 0, stream);
  if (err != cudaSuccess) return err;
  return launch_fixed_shape(work, n, batch, sms, B, hess, flag, itmax, state, stream);
}

}  // namespace tzg
