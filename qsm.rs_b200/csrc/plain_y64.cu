// Plain Y/Z passes in double precision (plain_passes.cuh).
#include "plain_passes.cuh"

namespace qsm {

template void run_yz_plain<double, -1, 1>(qsm_ctx*, const Fft3<double>&, const cplx_t<double>*, cplx_t<double>*, const int*);
template void run_yz_plain<double, +1, 1>(qsm_ctx*, const Fft3<double>&, const cplx_t<double>*, cplx_t<double>*, const int*);
template void run_yz_plain<double, -1, 2>(qsm_ctx*, const Fft3<double>&, const cplx_t<double>*, cplx_t<double>*, const int*);
template void run_yz_plain<double, +1, 2>(qsm_ctx*, const Fft3<double>&, const cplx_t<double>*, cplx_t<double>*, const int*);
template void tune_yz_fixed<double, -1, 1>(qsm_ctx*, const Fft3<double>&, const std::function<void()>&);
template void tune_yz_fixed<double, +1, 1>(qsm_ctx*, const Fft3<double>&, const std::function<void()>&);

}  // namespace qsm
