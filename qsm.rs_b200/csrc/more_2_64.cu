// Compile-time passes of the list QSM_FIXED_PLANS_MORE_2, double precision (more_plans.cuh).
#include "more_plans.cuh"

namespace qsm {

QSM_MORE_DEFINE(2)
QSM_MORE_INSTANTIATE(2, double)

}  // namespace qsm
