// Ragged backward (Abar for a batch of mixed orders): the planning of
// zgeev_ragged.cu, the Schur forms in 64-bit fixed point (zgeev_fixed_schur.cuh; orders of 5 and more, in
// classes of neighbouring orders, those above 32 on the caller's stream and the others beside them), then the
// persistent solver in backward mode. A translation unit of its own so that it compiles in parallel with the
// forward's.
#include <mutex>

#include "zgeev_ragged_work.cuh"

namespace tzg {

static cudaError_t ragged_schur_forms(int sms, int batch, RaggedPlan* plan, const RaggedArgs& a, cudaStream_t stream,
                                      const ForkJoin* fj) {
  const RaggedBatch B{a.A, a.offsets, a.eoff, nullptr};
  cfx* hess = reinterpret_cast<cfx*>(a.stage + a.region);
  cfx* q = reinterpret_cast<cfx*>(a.stage + 2 * a.region);
  const SchurDone done{a.stage, a.stage + 3 * a.region, a.gbar, a.eoff, nullptr, a.flag};
  const EigenvalueShifts shifts{a.lam, a.eoff};
  const bool two = fj != nullptr && fj->aux != nullptr;
  cudaError_t err = cudaSuccess;
  cudaStream_t side = stream;
  if (two) {
    if ((err = cudaEventRecord(fj->fork, stream)) != cudaSuccess) return err;
    if ((err = cudaStreamWaitEvent(fj->aux, fj->fork, 0)) != cudaSuccess) return err;
    side = fj->aux;
  }
  static const int kClass[6][2] = {{64, 49}, {48, 33}, {32, 25}, {24, 17}, {16, 9}, {8, 5}};
  const long long many = (long long)sms * 32;
  for (int pass = 0; pass < 2; ++pass)
    for (int c = 0; c < 6 && err == cudaSuccess; ++c) {
      const RaggedWork work{plan, a.sorted, kClass[c][0], kClass[c][1], true};
      const cudaStream_t s = kClass[c][0] > 32 ? stream : side;
      err = pass == 0 ? launch_schur_hess(work, kClass[c][0], batch, B, hess, q, many, s)
                      : launch_schur_qr(work, kClass[c][0], batch, shifts, done, hess, q, a.itmax_override,
                                        kGradDeflationUlps, many, s);
    }
  if (two) {  // also after a failed launch: the second stream rejoins the caller's
    const cudaError_t e1 = cudaEventRecord(fj->join, fj->aux);
    const cudaError_t e2 = cudaStreamWaitEvent(stream, fj->join, 0);
    if (err == cudaSuccess) err = e1 != cudaSuccess ? e1 : e2;
  }
  return err;
}

cudaError_t launch_ragged_backward(int lanes, int sms, int batch, const int* n, const long long* offsets,
                                   const long long* eig_offsets, long long total_elements, const double2* A,
                                   const double2* lam, const double2* gbar, double2* gA, void* work, char* flag,
                                   int itmax_override, cudaStream_t stream, int scaled_min_n, bool fixed,
                                   const ForkJoin* fj) {
  if (!(lanes == 0 || lanes == 1 || lanes == 2 || lanes == 4 || lanes == 8)) return cudaErrorInvalidValue;
  const RaggedLayout lay = ragged_layout(batch, total_elements, 4);
  double2* stage = reinterpret_cast<double2*>(static_cast<char*>(work) + lay.stage_off);
  RaggedPlan* plan;
  int* sorted;
  const long long* eo;
  cudaError_t err = ragged_prepare(lanes, sms, batch, n, offsets, eig_offsets, total_elements, lay, work, flag,
                                   stream, &plan, &sorted, &eo);
  if (err != cudaSuccess) return err;
  const RaggedArgs args{offsets, eo, A, nullptr, lam, gbar, gA, stage, total_elements, flag, sorted, itmax_override,
                        0, nullptr, nullptr, 0, fixed, scaled_min_n};
  if (fixed) {
    std::unique_lock<std::mutex> lock;
    if (fj != nullptr && fj->aux != nullptr) lock = std::unique_lock<std::mutex>(*fj->mu);
    if ((err = ragged_schur_forms(sms, batch, plan, args, stream, fj)) != cudaSuccess) return err;
  }
  return launch_ragged_kernel<true, false, kPhaseAll>(lanes, sms, plan, args, stream);
}

}  // namespace tzg
