// Instantiations of the stage kernels for orders 10, 11.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(10)
SDG_DEFINE_ORDER(11)
}  // namespace sdg
