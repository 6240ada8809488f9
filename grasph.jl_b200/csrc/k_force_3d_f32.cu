// k_force_3d_f32.cu — 3-D instantiations of the FP32-compensated pair sweep.
#include "k_sweep_f32.cuh"

namespace gc {

GC_DEFINE_FORCE_F32_TU(3, launch_force_3d_f32)

}  // namespace gc
