// Compile-time passes of the list QSM_FIXED_PLANS_MORE_0, double precision (more_plans.cuh).
#include "more_plans.cuh"

namespace qsm {

QSM_MORE_DEFINE(0)
QSM_MORE_INSTANTIATE(0, double)

}  // namespace qsm
