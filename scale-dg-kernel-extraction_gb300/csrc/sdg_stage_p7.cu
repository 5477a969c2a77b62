// Instantiations of the stage kernels for order 7.
#include "sdg_stage_order.cuh"

namespace sdg {
SDG_DEFINE_ORDER(7)
}  // namespace sdg
