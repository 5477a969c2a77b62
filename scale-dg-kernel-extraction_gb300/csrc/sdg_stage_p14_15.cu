// Instantiations of the stage kernels for orders 14, 15.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(14)
SDG_DEFINE_ORDER(15)
}  // namespace sdg
