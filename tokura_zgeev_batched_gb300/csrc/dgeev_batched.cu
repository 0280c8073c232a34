// Batched real eigenvalue-only entry points (LAPACK dgeev / sgeev with
// JOBVL = JOBVR = 'N'): tokura_dgeev_batched_gpu (FP64) and
// tokura_sgeev_batched_gpu (FP32 in and out, FP64 inside). Matrix j is
// column-major at A + j*n*n; its eigenvalues go to wr/wi[i + j*n] in LAPACK's
// convention (complex pairs adjacent, positive imaginary part first, exact
// conjugates). Same tiling as the complex plain kernel: a warp holds 32/L
// matrices of the batch, each on L lanes, staged tile-interleaved in work. Without settings of
// their own on the handle, matrices of order 3 and more are solved in 64-bit fixed point first (dgeev_fixed.cuh) and
// this kernel takes what that leaves. Measured (ms, FP64 alone and with fixed point): 1,000,000 of order 3 5.7 and 1.5,
// 250,000 of 8 8.6 and 3.9, 65,536 of 16 8.6 and 5.4, 10,000 of 32 10.1 and 5.9, 16,384 of 64 85.7 and 62.0.
#include <cstdint>
#include <type_traits>

#include "../../include/tokura_blas_ext.h"
#include "dgeev_fixed.cuh"
#include "dgeev_real.cuh"
#include "zgeev_fixed_launch.cuh"
#include "tokura_handle.h"

namespace tzg {

// kLeft: after the fixed-point kernels, only the matrices that they left (an instantiation of its own: with a run-time
// switch the FP64 calls were 3 to 5 % slower, 16,384 matrices of order 64 99.1 against 96.1 ms at two lanes).
template <int L, bool kBalance, bool kLeft, class T>
__global__ void __launch_bounds__(256) dgeev_plain_kernel(int n, int batch, const T* __restrict__ A,
                                                           T* __restrict__ wr, T* __restrict__ wi,
                                                           double* __restrict__ work, char* __restrict__ flag,
                                                           int itmax, int balance) {
  using Src = typename std::conditional<std::is_same<T, float>::value, SrcReal32, SrcReal64>::type;
  constexpr int TW = 32 / L;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long g0 = warp * TW;
  if (g0 >= batch) return;
  const int tw = (int)min((long long)TW, (long long)batch - g0);
  const int slot = lane / L;
  if (slot >= tw) return;
  const Group<L> G;
  const long long nn = (long long)n * n;
  const long long j = g0 + slot;
  if (kLeft && flag[j] != kLeftToFp64) return;  // group-uniform
  const RMatView M{work + g0 * nn + slot, n, tw};
  const int status = solve_real_matrix<L, kBalance>(Src{A + j * nn}, M, G, wr + j * n, wi + j * n, itmax, balance);
  if (G.rank == 0) flag[j] = (char)status;
}

template <int L, class T>
static void launch_real_l(unsigned blocks, int threads, cudaStream_t stream, int n, int batch, const T* A, T* wr,
                          T* wi, double* work, char* flag, int itmax, int balance, bool left_only) {
  if (left_only)
    dgeev_plain_kernel<L, false, true, T><<<blocks, threads, 0, stream>>>(n, batch, A, wr, wi, work, flag, itmax, 0);
  else if (balance != 0)
    dgeev_plain_kernel<L, true, false, T>
        <<<blocks, threads, 0, stream>>>(n, batch, A, wr, wi, work, flag, itmax, balance);
  else
    dgeev_plain_kernel<L, false, false, T><<<blocks, threads, 0, stream>>>(n, batch, A, wr, wi, work, flag, itmax, 0);
}

template <int L, class T>
static cudaError_t launch_real_hess(int n, int batch, const T* A, T* wr, T* wi, long long* work, char* flag,
                                    cudaStream_t stream) {
  constexpr int tw = L >= 32 ? 1 : 32 / L;
  real_hess_kernel<L, T><<<(unsigned)((batch + (long long)tw - 1) / tw), L > 32 ? L : 32, real_hess_shared<L>(n),
                           stream>>>(n, batch, A, wr, wi, work, flag, 1);
  return cudaGetLastError();
}

template <class T>
static cudaError_t launch_real_fixed(int n, int batch, int sms, const T* A, T* wr, T* wi, double* work0, char* flag,
                                     int itmax, cudaStream_t stream) {
  long long* const work = reinterpret_cast<long long*>(work0);
  const uintptr_t scratch = (reinterpret_cast<uintptr_t>(work + (long long)batch * real_words(n)) + 15) & ~(uintptr_t)15;
  const long long room = ((long long)(reinterpret_cast<uintptr_t>(work + (long long)batch * n * n) - scratch)) / 16;
  cudaError_t err;
  if (n <= 4)
    err = launch_real_hess<4>(n, batch, A, wr, wi, work, flag, stream);
  else if (n <= 8)
    err = launch_real_hess<8>(n, batch, A, wr, wi, work, flag, stream);
  else if (n <= 16)
    err = launch_real_hess<16>(n, batch, A, wr, wi, work, flag, stream);
  else if (n <= 32)
    err = launch_real_hess<32>(n, batch, A, wr, wi, work, flag, stream);
  else
    err = launch_real_hess<128>(n, batch, A, wr, wi, work, flag, stream);
  if (err != cudaSuccess) return err;
  const RealBatch B{work, wr, wi, std::is_same<T, float>::value, reinterpret_cast<cfx*>(scratch), room};
  return launch_fixed_shape(UniformWork{n, batch}, n, batch, sms, B, nullptr, flag, itmax, nullptr, stream);
}

template <class T>
static cudaError_t launch_real(const tokurablas_t* h, int n, int batch, const T* A, T* wr, T* wi, double* work,
                               char* flag, cudaStream_t stream) {
  const PlainConfig cfg = real_config_for(h, n, batch);
  const int L = cfg.lanes;
  const int tw = 32 / L;
  const long long warps = ((long long)batch + tw - 1) / tw;
  const int threads = cfg.threads;
  const long long blocks = (warps * 32 + threads - 1) / threads;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int itmax = h->itmax_override > 0 ? h->itmax_override : default_itmax(n);
  const int bal = h->balance_mode;
  const bool fixed = use_fixed_real(h, n);
  if (fixed) {
    const cudaError_t err = launch_real_fixed(n, batch, h->sm_count, A, wr, wi, work, flag, itmax, stream);
    if (err != cudaSuccess) return err;
  }
  switch (L) {
    case 1: launch_real_l<1>((unsigned)blocks, threads, stream, n, batch, A, wr, wi, work, flag, itmax, bal, fixed); break;
    case 2: launch_real_l<2>((unsigned)blocks, threads, stream, n, batch, A, wr, wi, work, flag, itmax, bal, fixed); break;
    case 4: launch_real_l<4>((unsigned)blocks, threads, stream, n, batch, A, wr, wi, work, flag, itmax, bal, fixed); break;
    case 8: launch_real_l<8>((unsigned)blocks, threads, stream, n, batch, A, wr, wi, work, flag, itmax, bal, fixed); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <class T>
static int real_entry(tokurablas_t* handle, int n, int batch_count, const T* A, T* wr, T* wi, double* work,
                      char* flag, cudaStream_t stream) {
  if (handle == nullptr) return -1;
  if (!(n > 0 && n <= TOKURA_ZGEEV_BATCHED_MAX_MATRIX_SIZE)) return -2;
  if (A == nullptr) return -3;
  if (wr == nullptr || wi == nullptr) return -4;
  if (work == nullptr) return -5;
  if (!(batch_count > 0)) return -6;
  if (flag == nullptr) return -7;
  return launch_real(handle, n, batch_count, A, wr, wi, work, flag, stream) == cudaSuccess ? 0 : 1;
}

}  // namespace tzg

extern "C" TOKURA_API size_t tokura_get_dgeev_workspacesize(int n, int batch_count) {
  if (!(n > 0 && n <= TOKURA_ZGEEV_BATCHED_MAX_MATRIX_SIZE)) return (size_t)-1;
  if (!(batch_count > 0)) return (size_t)-2;
  return sizeof(double) * (size_t)n * (size_t)n * (size_t)batch_count;
}

extern "C" TOKURA_API int tokura_dgeev_batched_gpu(tokurablas_t* handle, int n, int batch_count, const double* A,
                                                    double* wr, double* wi, double* work, char* flag,
                                                    cudaStream_t cudastream) {
  return tzg::real_entry(handle, n, batch_count, A, wr, wi, work, flag, cudastream);
}

extern "C" TOKURA_API int tokura_sgeev_batched_gpu(tokurablas_t* handle, int n, int batch_count, const float* A,
                                                    float* wr, float* wi, double* work, char* flag,
                                                    cudaStream_t cudastream) {
  return tzg::real_entry(handle, n, batch_count, A, wr, wi, work, flag, cudastream);
}
