// Instantiations of the stencil launcher: FP64 smoothing sweeps.
#include "stencil_launch.cuh"

namespace femh_engine {
#define INST(T, OUT, TI, TO, TB, TC)                                                                    \
  template void stencil<T, OUT, TI, TO, TB, TC>(femh_handle*, Level&, bool, const TI*, TO*, const TB*, \
                                                const TC*, double*, const CGState*, double);
INST(double, OUT_JACOBI, double, double, double, double)
INST(double, OUT_JACOBI_DOT, double, double, double, double)
INST(double, OUT_RESID, double, double, double, double)
}  // namespace femh_engine
