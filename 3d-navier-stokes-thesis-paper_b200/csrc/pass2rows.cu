// pass2rows.cu -- launcher of the row-per-thread substep kernel
// (pass2rows.cuh).
#include "pass2rows.cuh"

namespace cfd {

template <typename S>
__global__ void __launch_bounds__(256) k_rhs_rows(RhsRowsLaunch a) {
  k_rhs_rows_block<S>(blockIdx.x, a);
}

// Batched launch over a member table (the ensemble mode): member m of a class
// of identical grids takes blocks m*gx ... m*gx + gx - 1 and reads its
// arguments from its launch record in device memory.
template <typename S>
__global__ void __launch_bounds__(256) k_rhs_rows_b(const RhsRowsLaunch* __restrict__ tab, unsigned gx) {
  const unsigned m = blockIdx.x / gx;
  k_rhs_rows_block<S>((int)(blockIdx.x - m * gx), tab[m]);
}

int rhs_rows_launch(bool f32, const RhsRowsLaunch& a) { return rhs_rows_launch_batch(f32, a, nullptr, 1); }

int rhs_rows_launch_batch(bool f32, const RhsRowsLaunch& a, const RhsRowsLaunch* tab, int nmem) {
  if (nmem < 1 || a.g.ny1 > 256) return -1;
  const int low = a.nlist + (a.mean ? 1 : 0);
  const unsigned gx = (unsigned)(low + a.nfast);
  if (gx == 0) return 0;
  const int nt = rhs_rows_threads(a.g.ny1);
  const size_t sm = rhs_rows_smem(a.g.ny1);
  if (tab && f32) k_rhs_rows_b<float><<<gx * nmem, nt, sm, a.st>>>(tab, gx);
  else if (tab) k_rhs_rows_b<double><<<gx * nmem, nt, sm, a.st>>>(tab, gx);
  else if (f32) launch_chained(a.pdl, k_rhs_rows<float>, dim3(gx), dim3(nt), sm, a.st, a);
  else launch_chained(a.pdl, k_rhs_rows<double>, dim3(gx), dim3(nt), sm, a.st, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace cfd
