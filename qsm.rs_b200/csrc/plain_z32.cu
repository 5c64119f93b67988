// Multiplier Z pass in single precision (plain_passes.cuh).
#include "plain_passes.cuh"

namespace qsm {

template void run_z_fused_m<float>(qsm_ctx*, const Fft3<float>&, const cplx_t<float>*, cplx_t<float>*, const float*, const int*);
template void tune_z_fused_m<float>(qsm_ctx*, const Fft3<float>&, const std::function<void()>&);

}  // namespace qsm
