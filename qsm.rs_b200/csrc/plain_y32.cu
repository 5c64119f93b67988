// Plain Y/Z passes in single precision (plain_passes.cuh).
#include "plain_passes.cuh"

namespace qsm {

template void run_yz_plain<float, -1, 1>(qsm_ctx*, const Fft3<float>&, const cplx_t<float>*, cplx_t<float>*, const int*);
template void run_yz_plain<float, +1, 1>(qsm_ctx*, const Fft3<float>&, const cplx_t<float>*, cplx_t<float>*, const int*);
template void run_yz_plain<float, -1, 2>(qsm_ctx*, const Fft3<float>&, const cplx_t<float>*, cplx_t<float>*, const int*);
template void run_yz_plain<float, +1, 2>(qsm_ctx*, const Fft3<float>&, const cplx_t<float>*, cplx_t<float>*, const int*);
template void tune_yz_fixed<float, -1, 1>(qsm_ctx*, const Fft3<float>&, const std::function<void()>&);
template void tune_yz_fixed<float, +1, 1>(qsm_ctx*, const Fft3<float>&, const std::function<void()>&);

}  // namespace qsm
