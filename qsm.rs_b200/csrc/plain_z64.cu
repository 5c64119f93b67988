// Multiplier Z pass in double precision (plain_passes.cuh).
#include "plain_passes.cuh"

namespace qsm {

template void run_z_fused_m<double>(qsm_ctx*, const Fft3<double>&, const cplx_t<double>*, cplx_t<double>*, const double*, const int*);
template void tune_z_fused_m<double>(qsm_ctx*, const Fft3<double>&, const std::function<void()>&);

}  // namespace qsm
