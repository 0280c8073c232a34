// tokuraDebugAttach: attaches a device DebugRecord (zgeev_debug.cuh) to every
// translation unit's kernels in the bounds-checked build; the release build
// exports the same entry point and returns -2. tokuraDebugChecks: the accesses
// that Checked pointers have checked so far.
#include <vector>

#include "../../include/tokura_blas_ext.h"
#include "zgeev_debug.cuh"

namespace tzg {
#ifdef TOKURA_DEBUG_BOUNDS
struct DebugUnit {
  DebugAttachFn attach;
  DebugChecksFn checks;
};
static std::vector<DebugUnit>& debug_registry() {
  static std::vector<DebugUnit> units;
  return units;
}
void debug_register(DebugAttachFn attach, DebugChecksFn checks) { debug_registry().push_back({attach, checks}); }
#endif
}  // namespace tzg

extern "C" TOKURA_API int tokuraDebugAttach(void* record) {
#ifdef TOKURA_DEBUG_BOUNDS
  for (const tzg::DebugUnit& unit : tzg::debug_registry())
    if (unit.attach(static_cast<tzg::DebugRecord*>(record)) != cudaSuccess) return 1;
  return 0;
#else
  (void)record;
  return -2;
#endif
}

extern "C" TOKURA_API int tokuraDebugChecks(unsigned long long* checks) {
#ifdef TOKURA_DEBUG_BOUNDS
  if (checks == nullptr) return -1;
  *checks = 0;
  for (const tzg::DebugUnit& unit : tzg::debug_registry()) {
    unsigned long long n = 0;
    if (unit.checks(&n) != cudaSuccess) return 1;
    *checks += n;
  }
  return 0;
#else
  (void)checks;
  return -2;
#endif
}
