// Instantiations of the stencil launcher: FP32 operator and residual.
#include "stencil_launch.cuh"

namespace femh_engine {
#define INST(T, OUT, TI, TO, TB, TC)                                                                    \
  template void stencil<T, OUT, TI, TO, TB, TC>(femh_handle*, Level&, bool, const TI*, TO*, const TB*, \
                                                const TC*, double*, const CGState*, double);
INST(float, OUT_APPLY, float, float, float, float)
INST(float, OUT_RESID, float, float, float, float)
INST(float, OUT_APPLY_DOT, float, float, float, float)
INST(float, OUT_APPLY_DOT, __nv_bfloat16, float, float, float)
}  // namespace femh_engine
