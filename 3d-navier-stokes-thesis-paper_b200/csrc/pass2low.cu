// pass2low.cu -- launcher of the FP64 substep kernel of the mean mode and the
// mixed path's |k| < 4 list (pass2low.cuh).
#include "pass2low.cuh"

namespace cfd {

template <typename S>
__global__ void __launch_bounds__(256) k_rhs_low(RhsLowLaunch a) {
  k_rhs_low_body<S>(blockIdx.x, a);
}

// Batched launch over a member table (the ensemble mode): member m of a class
// of identical grids takes blocks m*gx ... m*gx + gx - 1 and reads its
// arguments from its launch record in device memory.
template <typename S>
__global__ void __launch_bounds__(256) k_rhs_low_b(const RhsLowLaunch* __restrict__ tab, unsigned gx) {
  const unsigned m = blockIdx.x / gx;
  k_rhs_low_body<S>((int)(blockIdx.x - m * gx), tab[m]);
}

int rhs_low_launch(bool f32, const RhsLowLaunch& a) { return rhs_low_launch_batch(f32, a, nullptr, 1); }

int rhs_low_launch_batch(bool f32, const RhsLowLaunch& a, const RhsLowLaunch* tab, int nmem) {
  if (nmem < 1 || a.g.ny1 > 256) return -1;
  const unsigned gx = (unsigned)(a.nlist + (a.mean ? 1 : 0));
  if (gx == 0) return 0;
  const int nt = rhs_low_threads(a.g.ny1);
  const size_t sm = rhs_low_smem(a.g.ny1);
  if (tab && f32) k_rhs_low_b<float><<<gx * nmem, nt, sm, a.st>>>(tab, gx);
  else if (tab) k_rhs_low_b<double><<<gx * nmem, nt, sm, a.st>>>(tab, gx);
  else if (f32) k_rhs_low<float><<<gx, nt, sm, a.st>>>(a);
  else k_rhs_low<double><<<gx, nt, sm, a.st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace cfd
