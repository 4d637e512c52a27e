// rve_modes_inst_cube_per.cu -- instantiations of the element-mode batch kernel
// (rve_modes_kernel.cuh) for cubic elements, periodic conditions.
#include "rve_modes_kernel.cuh"

namespace sp {
#define SP_MODES_DEFINE(V, NT, MINB, QS) \
  template __global__ void k_modes<V, NT, MINB, true, QS, true>(ModesParams);
SP_MODES_CLASSES(SP_MODES_DEFINE, F2)
}  // namespace sp
