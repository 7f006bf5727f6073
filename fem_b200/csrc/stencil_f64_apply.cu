// Instantiations of the stencil launcher: FP64 operator, search directions of every storage type.
#include "stencil_launch.cuh"

namespace femh_engine {
#define INST(T, OUT, TI, TO, TB, TC)                                                                    \
  template void stencil<T, OUT, TI, TO, TB, TC>(femh_handle*, Level&, bool, const TI*, TO*, const TB*, \
                                                const TC*, double*, const CGState*, double);
INST(double, OUT_APPLY, double, double, double, double)
INST(double, OUT_APPLY_DOT, double, double, double, double)
INST(double, OUT_APPLY_DOT, float, double, double, double)
INST(double, OUT_APPLY_DOT, __nv_bfloat16, double, double, double)
}  // namespace femh_engine
