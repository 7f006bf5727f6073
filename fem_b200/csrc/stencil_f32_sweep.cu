// Instantiations of the stencil launcher: FP32 smoothing sweeps.
#include "stencil_launch.cuh"

namespace femh_engine {
#define INST(T, OUT, TI, TO, TB, TC)                                                                    \
  template void stencil<T, OUT, TI, TO, TB, TC>(femh_handle*, Level&, bool, const TI*, TO*, const TB*, \
                                                const TC*, double*, const CGState*, double);
INST(float, OUT_JACOBI, float, float, float, float)
INST(float, OUT_JACOBI_DOT, float, float, float, float)
}  // namespace femh_engine
