// Ragged forward in 64-bit fixed point (zgeev_fixed.cuh): the planner's bins (matrices sorted by order) are
// cut into classes of neighbouring orders, each with the launch shapes of a uniform batch of its largest order:
//   caller's stream: [planning] --fork-- [orders 49..64, 33..48] --join-- [FP64: what was left]
//   second stream:                 \---- [orders 25..32 .. 2..4] --/
// The classes above n = 32 keep their matrices in the workspace and the others in shared memory, so the two
// streams' kernels fit on an SM together, and one's last, half-empty wave is filled by the other. In large batches the waves are many and what the two evict from each other's caches costs more: all on the caller's
// stream. The limit, 100 matrices per SM of any order (15,200 on 152 SMs), lies between measurements that do not agree on one: orders
// in U{1..64}, two streams and one, 1,000 matrices 9.6 and 12.0 ms, 4,000 13.0 and 14.2, 9,000 22.7 and 20.3, 13,000 24.0
// and 26.2, 20,000 45.4 and 37.2, 60,000 117 and 100, 200,000 397 and 319; other ranges of orders were not measured.
#include "zgeev_ragged_work.cuh"

namespace tzg {

cudaError_t ragged_launch_fixed(int sms, int batch, RaggedPlan* plan, const RaggedArgs& args, cudaStream_t stream,
                                const ForkJoin* fj) {
  const RaggedBatch B{args.A, args.offsets, args.eoff, args.eig};
  cfx* hess = reinterpret_cast<cfx*>(args.stage);
  const int itmax = args.itmax_override;
  const bool two = batch < sms * 100 && fj != nullptr && fj->aux != nullptr;
  cudaError_t err = cudaSuccess;
  cudaStream_t side = stream;
  if (two) {
    if ((err = cudaEventRecord(fj->fork, stream)) != cudaSuccess) return err;
    if ((err = cudaStreamWaitEvent(fj->aux, fj->fork, 0)) != cudaSuccess) return err;
    side = fj->aux;
  }
  const long long many = (long long)sms * 32;
  auto fits = [&](int lanes, int warps) { return (long long)batch * lanes <= many * warps; };
#define TZG_HESS(NHI, NLO, L, STREAM)                                                                       \
  if (err == cudaSuccess)                                                                                   \
    err = launch_fixed_hess<L>(RaggedWork{plan, args.sorted, NHI, NLO}, NHI, batch, B, hess, args.flag, args.state, \
                               many, STREAM)
#define TZG_QR(NHI, NLO, L, T, G, BLOCKS, STREAM)                                                             \
  if (err == cudaSuccess)                                                                                     \
    err = launch_fixed_qr<L, T, G>(RaggedWork{plan, args.sorted, NHI, NLO}, NHI, batch, B, hess, args.flag, itmax, \
                                   args.state, BLOCKS, STREAM)
  TZG_HESS(64, 49, 128, stream);
  TZG_HESS(48, 33, 128, stream);
  TZG_QR(64, 49, 32, 2, true, (long long)sms * 24, stream);
  // Orders 33 to 48 at 32 and 16 lanes: 20,000 orders in U{1..64} 37.2 and 38.6 ms, 30,000 53.4 and 52.7, 60,000 102.3 and
  // 99.5, 200,000 331 and 319 (more lanes while the class is a wave or two).
  if (batch < sms * 200) {
    TZG_QR(48, 33, 32, 2, true, (long long)sms * 24, stream);
  } else {
    TZG_QR(48, 33, 16, 4, true, (long long)sms * 14, stream);
  }
  TZG_HESS(32, 25, 32, side);
  TZG_HESS(24, 17, 32, side);
  TZG_HESS(16, 9, 16, side);
  TZG_HESS(8, 5, 8, side);
  TZG_HESS(4, 2, 4, side);
  if (fits(8, 16)) {  // few matrices: as the small uniform batches
    TZG_QR(32, 25, 32, 1, false, many, side);
    TZG_QR(24, 17, 32, 1, false, many, side);
    TZG_QR(16, 9, 16, 1, false, many, side);
    TZG_QR(8, 5, 8, 1, false, many, side);
    TZG_QR(4, 2, 4, 1, false, many, side);
  } else {
    TZG_QR(32, 25, 16, 2, false, many, side);
    TZG_QR(24, 17, 8, 4, false, many, side);
    TZG_QR(16, 9, 4, 4, false, many, side);
    TZG_QR(8, 5, 2, 4, false, many, side);
    TZG_QR(4, 2, 1, 4, false, many, side);
  }
#undef TZG_HESS
#undef TZG_QR
  if (two) {  // also after a failed launch: the second stream rejoins the caller's
    const cudaError_t e1 = cudaEventRecord(fj->join, fj->aux);
    const cudaError_t e2 = cudaStreamWaitEvent(stream, fj->join, 0);
    if (err == cudaSuccess) err = e1 != cudaSuccess ? e1 : e2;
  }
  return err;
}

}  // namespace tzg
