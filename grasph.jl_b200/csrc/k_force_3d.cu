// k_force_3d.cu — 3-D instantiations of the FP64 sweeps: the window sweep
// of the fluid and stress functors, the buffered one of the others.
// Compiled with -fmad=false (fused operations are explicit fma()).
#include "k_sweep_f64.cuh"

namespace gc {

GC_DEFINE_FORCE_F64_TU(3, launch_force_3d_f64)

}  // namespace gc
