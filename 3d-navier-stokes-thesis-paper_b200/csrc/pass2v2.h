// pass2v2.h -- launch interface of the v2 RK substep kernel.
#pragma once
#include <cuda_runtime.h>

#include "pass1.cuh"
#include "pass2.cuh"

namespace cfd {

struct Rhs2Launch {
  void *vel, *cru, *prs;
  const void *cbc_top, *cbc_bot;
  Geom g;
  GridDev gd;
  const DevScalars* sc;
  RkTab rkt;
  int rk;
  double re;
  const int* wlist;
  int nlist;
  int warps;   // warps per block
  int lanes;   // lanes per wavenumber: 32, or 16 or 8 (FP32 only)
  const void* tbl;   // coefficient table of rhs2_table for these lanes
  cudaStream_t st;
};

// 0 on success, -1 unsupported size, -2 launch error
int rhs2_launch(bool f32, const Rhs2Launch& a);
// the same kernel for nmem members of one grid in one launch: tab is the
// members' launch records in device memory, a the first member's (host)
// copy, which sets the launch shape and stream
int rhs2_launch_batch(bool f32, const Rhs2Launch& a, const Rhs2Launch* tab, int nmem);

// the mean mode and, in mixed precision, the |k| < 4 list, in FP64 over the
// stored state (k_rhs_low, pass2low.cuh)
struct RhsLowLaunch {
  void *vel, *cru, *prs;
  double2 *mvel64, *mcru64;   // FP64 mean columns (mixed), or null
  const void *cbc_top, *cbc_bot;
  Geom g;
  GridDev gd;
  DevScalars* sc;
  double* d_um_dy;
  RkTab rkt;
  int rk;
  double re, beta;
  int fix_mass;
  int mean;                   // 1: this rank holds the mean mode
  const int* wlist;
  int nlist;
  cudaStream_t st;
};
int rhs_low_launch(bool f32, const RhsLowLaunch& a);
int rhs_low_launch_batch(bool f32, const RhsLowLaunch& a, const RhsLowLaunch* tab, int nmem);
bool rhs2_supported(int ny1);
// the lane-major grid-coefficient table the kernel reads (host side)
size_t rhs2_table_bytes(bool f32, int ny1, int lanes);
void rhs2_table(bool f32, int ny, int lanes, const double* dh, const double* dn, const double* d2h,
                const double* d2n, void* out);

}  // namespace cfd
