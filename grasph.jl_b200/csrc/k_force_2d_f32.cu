// k_force_2d_f32.cu — 2-D instantiations of the FP32-compensated pair sweep.
#include "k_sweep_f32.cuh"

namespace gc {

GC_DEFINE_FORCE_F32_TU(2, launch_force_2d_f32)

}  // namespace gc
