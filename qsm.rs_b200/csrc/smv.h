// Spherical-mean-value kernels: k-space multipliers of the normalised sphere and mask
// erosion by it (src/kernels/smv.rs:19-105), shared by the background-removal solvers.
#pragma once

#include <vector>

#include "launch.cuh"

namespace qsm {

// Voxels of the normalised sphere of `radius` mm at wrap-centred coordinates: for each
// pair of offsets (y, z) >= 0 the half-width of the x run inside, -1 where none.
struct SmvSphere {
  int nx, ny, nz;
  int dy, dz;             // largest offsets with voxels inside
  std::vector<int> half;  // [dz + 1][dy + 1]
  double r2;              // radius^2
  double total;           // voxels inside
};
SmvSphere smv_sphere(const GridDims& d, double radius);

// Half-spectrum multiplier arrays built from S = FFT(sphere kernel), evaluated in double.
enum SmvMult {
  kSmvS = 0,          // S
  kSmvOneMinusS = 1,  // 1 - S
  kSmvDeconv = 2      // 1 / (1 - S), 0 where |1 - S| < threshold
};
template <typename T>
void smv_multiplier(qsm_ctx* ctx, const Fft3<T>& f, const SmvSphere& s, SmvMult kind, double threshold, T* out);

// 1 - S in single precision from the transform of the sphere's image.  Its last bits differ
// from the cosine sums', which flips a rounding to single precision somewhere in most large
// spectra: for callers whose map must keep its roundings (restrict_forms).
void smv_one_minus_transform(qsm_ctx* ctx, const GridDims& d, const SmvSphere& s, float* out);

// Erosion by several spheres (mean of the mask over the sphere > delta), largest first:
// first[i] = index of the first sphere that keeps voxel i, 255 when none does.  At most
// 254 spheres.
void smv_erode_first(qsm_ctx* ctx, const GridDims& d, const uint8_t* mask, const std::vector<SmvSphere>& spheres,
                     double delta, uint8_t* first);

}  // namespace qsm
