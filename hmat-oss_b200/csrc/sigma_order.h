// The order in which the truncation kernels take singular values: descending, ties by index, NaN
// before every number.  Total, so the positions counted with it are a permutation whatever the
// values are: they index shared memory before the leaf's failure to converge is looked at.
#pragma once

#ifdef __CUDACC__
#define HB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define HB_HOST_DEVICE inline
#endif

namespace hmatb200 {

// Whether value a at index i comes before value b at index j (i != j).
HB_HOST_DEVICE bool sigma_before(double a, int i, double b, int j) {
  const bool nan_a = a != a, nan_b = b != b;
  if (nan_a != nan_b) return nan_a;
  return a > b || (!(a < b) && i < j);
}

}  // namespace hmatb200
