// Instantiations of the stage kernels for orders 1, 2, 3, 4.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(1)
SDG_DEFINE_ORDER(2)
SDG_DEFINE_ORDER(3)
SDG_DEFINE_ORDER(4)
}  // namespace sdg
