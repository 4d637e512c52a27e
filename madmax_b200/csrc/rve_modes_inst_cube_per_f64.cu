// rve_modes_inst_cube_per_f64.cu -- instantiations of the element-mode batch kernel
// (rve_modes_kernel.cuh) for cubic elements, periodic conditions, FP64.
#include "rve_modes_kernel.cuh"

namespace sp {
#define SP_MODES_DEFINE(V, NT, MINB, ON, PER) \
  template __global__ void k_modes<V, NT, MINB, true, ON, PER>(ModesParams);
SP_MODES_CLASSES(SP_MODES_DEFINE, double, true)
SP_MODES_PERIODIC(SP_MODES_DEFINE, double)
}  // namespace sp
