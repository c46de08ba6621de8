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
  int pdl;           // launched as the dependent of the kernel before it
  cudaStream_t st;
};

// 0 on success, -1 unsupported size, -2 launch error
int rhs2_launch(bool f32, const Rhs2Launch& a);
// the mixed path's |k| < 4 list beside the learned closure (see
// step_keeps_sums in capi.cu): FP64 arithmetic over FP32 storage, tbl the
// FP64 table for 32 lanes
int rhs2_launch_prec(const Rhs2Launch& a);
// the same kernel for nmem members of one grid in one launch: tab is the
// members' launch records in device memory, a the first member's (host)
// copy, which sets the launch shape and stream
int rhs2_launch_batch(bool f32, const Rhs2Launch& a, const Rhs2Launch* tab, int nmem);

// the mean mode beside the learned closure (k_rhs_mean2)
struct RhsMeanLaunch {
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
  const double* tbl64;        // FP64 coefficient table for 32 lanes
  cudaStream_t st;
};
int rhs_mean2_launch(bool f32, const RhsMeanLaunch& a);
// one block per wavenumber (k_rhs_rows, pass2rows.cuh): the mean mode and, in
// mixed precision, the |k| < 4 list in FP64 over the stored state; on small
// grids the fast list too
struct RhsRowsLaunch {
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
  int advance;                // the mean mode's block adds dt to t_total
  const int* wlist;           // FP64 list
  int nlist;
  double2 *lvel64, *lcru64, *lprs64;   // its FP64 columns (nlist x 3 x ny1 and nlist x ny1)
  const double2* jet64;       // the list's wall-normal wall values [bot, top][nlist], or null (cbc)
  const int* wfast;           // the fast list, nfast 0 where k_rhs2 takes it
  int nfast;
  int pdl;
  cudaStream_t st;
};
int rhs_rows_launch(bool f32, const RhsRowsLaunch& a);
int rhs_rows_launch_batch(bool f32, const RhsRowsLaunch& a, const RhsRowsLaunch* tab, int nmem);
bool rhs2_supported(int ny1);
// the lane-major grid-coefficient table the kernel reads (host side)
size_t rhs2_table_bytes(bool f32, int ny1, int lanes);
void rhs2_table(bool f32, int ny, int lanes, const double* dh, const double* dn, const double* d2h,
                const double* d2n, void* out);

}  // namespace cfd
