// Instantiations of the stage kernels for orders 5, 6.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(5)
SDG_DEFINE_ORDER(6)
}  // namespace sdg
