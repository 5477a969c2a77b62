// Instantiations of the stage kernels for orders 12, 13.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(12)
SDG_DEFINE_ORDER(13)
}  // namespace sdg
