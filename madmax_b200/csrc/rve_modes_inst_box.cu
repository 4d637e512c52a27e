// rve_modes_inst_box.cu -- instantiations of the element-mode batch kernel
// (rve_modes_kernel.cuh) for box elements.
#include "rve_modes_kernel.cuh"

namespace sp {
#define SP_MODES_DEFINE(V, NT, MINB, ON, PER) \
  template __global__ void k_modes<V, NT, MINB, false, ON, PER>(ModesParams);
SP_MODES_CLASSES(SP_MODES_DEFINE, F2, false)
SP_MODES_AFFINE(SP_MODES_DEFINE, F2)
}  // namespace sp
