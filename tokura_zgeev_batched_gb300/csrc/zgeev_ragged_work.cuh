// Ragged batches as the work and batch of the fixed-point kernels (zgeev_fixed_launch.cuh).
#pragma once

#include "zgeev_fixed_launch.cuh"
#include "zgeev_ragged.cuh"

namespace tzg {

// Matrices of orders nhi down to nlo; a tile holds matrices of one order.
struct RaggedWork {
  const RaggedPlan* plan;
  const int* sorted;
  int nhi, nlo;
  bool square = false;  // n^2 entries apart in the workspace
  __device__ __forceinline__ bool tile(long long t, int tw, int slot, FixedTile& out) const {
    if (plan->overflow) return false;
    // A class without matrices: two loads instead of one for each of its orders.
    const RaggedBin &top = plan->bins[kMaxN - nhi], &low = plan->bins[kMaxN - nlo];
    if (low.first + low.count == top.first) return false;
    for (int nb = nhi; nb >= nlo; --nb) {
      const RaggedBin& bin = plan->bins[kMaxN - nb];
      const int tiles = (bin.count + tw - 1) / tw;
      if (t < tiles) {
        const int p = (int)t * tw;
        out.n = nb;
        out.count = min(tw, bin.count - p);
        out.j = slot < out.count ? sorted[bin.first + p + slot] : 0;
        out.where = bin.stage + (long long)p * (square ? nb * nb : hess_stride(nb));
        out.origin = bin.stage;
        out.total = bin.count;
        out.pos = p;
        out.width = 32 / bin.lanes;
        return true;
      }
      t -= tiles;
    }
    return false;
  }
};

struct RaggedBatch {
  const double2* A;
  const long long* offsets;
  const long long* eoff;
  double2* eig;
  __device__ __forceinline__ bool valid(long long) const { return true; }
  __device__ __forceinline__ SrcContig src(long long j) const { return SrcContig{A + offsets[j]}; }
  __device__ __forceinline__ double2* out(long long j, int) const { return eig + eoff[j]; }
};

}  // namespace tzg
