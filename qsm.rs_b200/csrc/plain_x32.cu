// Plain X passes in single precision (plain_passes.cuh).
#include "plain_passes.cuh"

namespace qsm {

template bool x_plain_r2c<float>(qsm_ctx*, const Fft3<float>&, const float*, cplx_t<float>*, const int*);
template bool x_plain_c2r<float>(qsm_ctx*, const Fft3<float>&, const cplx_t<float>*, float*, float, const int*);

}  // namespace qsm
