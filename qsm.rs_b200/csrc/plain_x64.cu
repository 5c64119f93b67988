// Plain X passes in double precision (plain_passes.cuh).
#include "plain_passes.cuh"

namespace qsm {

template bool x_plain_r2c<double>(qsm_ctx*, const Fft3<double>&, const double*, cplx_t<double>*, const int*);
template bool x_plain_c2r<double>(qsm_ctx*, const Fft3<double>&, const cplx_t<double>*, double*, double, const int*);

}  // namespace qsm
