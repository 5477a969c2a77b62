// Instantiations of the stage kernels for orders 8, 9.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(8)
SDG_DEFINE_ORDER(9)
}  // namespace sdg
