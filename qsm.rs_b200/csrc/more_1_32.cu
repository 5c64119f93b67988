// Compile-time passes of the list QSM_FIXED_PLANS_MORE_1, single precision (more_plans.cuh).
#include "more_plans.cuh"

namespace qsm {

QSM_MORE_DEFINE(1)
QSM_MORE_INSTANTIATE(1, float)

}  // namespace qsm
