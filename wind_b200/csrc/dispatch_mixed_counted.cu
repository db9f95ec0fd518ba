// dispatch_mixed_counted.cu -- instantiations of k_mixed that stage their teams'
// systems by counting (mixed_counted).
#include "api_internal.h"
#include "mixed_kernel.cuh"

namespace wind {

MixedFn mixed_fn_counted(int method, int ctrl, int solver) { return mixed_fn<true>(method, ctrl, solver); }

}  // namespace wind
