// Compile-time passes of the list QSM_FIXED_PLANS_MORE_3, double precision (more_plans.cuh).
#include "more_plans.cuh"

namespace qsm {

QSM_MORE_DEFINE(3)
QSM_MORE_INSTANTIATE(3, double)

}  // namespace qsm
