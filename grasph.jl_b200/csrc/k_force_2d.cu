// k_force_2d.cu — 2-D instantiations of the FP64 sweeps: the window sweep
// of the fluid and stress functors, the buffered one of the others.
// Compiled with -fmad=false (fused operations are explicit fma()).
#include "k_sweep_f64.cuh"

namespace gc {

GC_DEFINE_FORCE_F64_TU(2, launch_force_2d_f64)

}  // namespace gc
