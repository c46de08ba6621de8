// pass2rows.cuh -- the RK3/Crank-Nicolson substep of PFC/pass2.f90:184-352
// with one block per wavenumber and one thread per row of its columns:
//   - for the mean mode with its constant-mass-flux pressure gradient
//     (PFC/pass2.f90:217-263, 356-375) and, in mixed precision, for |k| < 4,
//     whose pressure problem is ill-conditioned in FP32 on the stretched grid;
//   - for all the others where the grid is so small that the main kernel
//     (k_rhs2) would not fill the GPU.
// The arithmetic is FP64 over the stored state; in mixed precision the mean
// mode and the FP64 list keep FP64 columns beside their FP32 ones.
//
// What bounds these cases is the length of one block's chain, and a chain
// executed once pays for every instruction it fetches: k_rhs2's form, several
// rows per lane of a warp, unrolls to code that no instruction cache holds
// (55 us in FP64 for 49 wavenumbers of 194 rows, mean mode 36 us; 12 us for
// both together here).  With a row per thread the tridiagonal systems are
// solved by parallel cyclic reduction in a rolled loop over shared memory --
// log2(rows) steps, more operations but a chain of a few thousand cycles in
// little code; the u/w system (two right-hand sides) and the v system go
// through one loop.
#pragma once
#include "cfd_common.cuh"
#include "pass1.cuh"
#include "pass2.cuh"
#include "pass2v2.cuh"
#include "pass2v2.h"

namespace cfd {

// shared memory per row: two copies of the reduction's couplings (six values)
// and right-hand sides (three complex values); the staged columns (four
// complex values) share the first copy
__host__ __device__ __forceinline__ int rhs_rows_threads(int n1) { return (n1 + 31) & ~31; }
__host__ __device__ __forceinline__ size_t rhs_rows_smem(int n1) {
  return (size_t)rhs_rows_threads(n1) * 2 * 12 * sizeof(double);
}

// Parallel cyclic reduction of NM tridiagonal systems over the block's rows:
// row j of system m is x_j = a[m] x_{j-1} + c[m] x_{j+1} + f (divided by its
// diagonal; a = 0 in the first and c = 0 in the last row), a, c >= 0, with
// the diagonal's excess e[m] = 1 - a[m] - c[m] >= 0; right-hand side r
// belongs to system r < NR - 1 ? 0 : NM - 1.  The solutions come back in f.
// The pressure rows' excess is k^2 h^2 beside one, and a reduced diagonal
// formed as 1 - a c_l - c a_u would lose it (4 times the first solver's error
// at 256 rows); carried as a value of its own (as in the elimination of
// Grassmann, Taksar and Heyman) every update adds positive terms only.
// buf: two halves of NM*3 real and NR complex values per thread.  Every
// thread of the block calls it, rows past the system as identity rows
// (a = c = 0, e = 1).
template <typename T, int NM, int NR>
__device__ __forceinline__ void pcr_rows(T (&a)[NM], T (&c)[NM], T (&e)[NM], cplx_t<T> (&f)[NR], int n, void* buf) {
  using C = cplx_t<T>;
  const int j = threadIdx.x, nt = blockDim.x;
  const T tiny = (T)1e-30;   // couplings that no longer reach the last bit
  T* const base = reinterpret_cast<T*>(buf);
  const int half = nt * (3 * NM + 2 * NR + (NM & 1));   // (complex values stay aligned)
  int h = 0;
#pragma unroll 1
  for (int s = 1; s < n; s <<= 1, h ^= 1) {
    C* const fs = reinterpret_cast<C*>(base + h * half);
    T* const ac = reinterpret_cast<T*>(fs + NR * nt);
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      ac[(3 * m) * nt + j] = a[m];
      ac[(3 * m + 1) * nt + j] = c[m];
      ac[(3 * m + 2) * nt + j] = e[m];
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) fs[r * nt + j] = f[r];
    // decoupled rows (a viscous step couples a row to few neighbours): done
    bool open = false;
#pragma unroll
    for (int m = 0; m < NM; ++m) open = open || a[m] > tiny || c[m] > tiny;
    if (!__syncthreads_or(open)) break;
    // a coupling past an end is zero: the clamped neighbour's values drop out
    const int l = max(j - s, 0), u = min(j + s, nt - 1);
    T rb[NM], fa[NM], fc[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const T al = ac[(3 * m) * nt + l], el = ac[(3 * m + 2) * nt + l];
      const T cu = ac[(3 * m + 1) * nt + u], eu = ac[(3 * m + 2) * nt + u];
      fa[m] = a[m];
      fc[m] = c[m];
      // 1 - a c_l - c a_u with c_l = 1 - a_l - e_l and a_u = 1 - c_u - e_u
      rb[m] = rcpv<T>(e[m] + fa[m] * (el + al) + fc[m] * (eu + cu));
      e[m] = (e[m] + fa[m] * el + fc[m] * eu) * rb[m];
      a[m] = fa[m] * al * rb[m];
      c[m] = fc[m] * cu * rb[m];
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int m = r < NR - 1 ? 0 : NM - 1;
      const C fl = fs[r * nt + l], fu = fs[r * nt + u];
      f[r] = mk<C>((f[r].x + fa[m] * fl.x + fc[m] * fu.x) * rb[m], (f[r].y + fa[m] * fl.y + fc[m] * fu.y) * rb[m]);
    }
  }
  __syncthreads();
}

// second difference at row j of an n-row column s (end rows copy their
// neighbours' stencil), coefficients d2[3 j ..]
template <typename T>
__device__ __forceinline__ cplx_t<T> d2_of_row(const cplx_t<T>* s, const double* __restrict__ d2, int j, int n) {
  using C = cplx_t<T>;
  const int j0 = j == 0 ? 1 : (j == n - 1 ? n - 2 : j);
  const T d1 = (T)__ldg(d2 + 3 * j), d0 = (T)__ldg(d2 + 3 * j + 1), d3 = (T)__ldg(d2 + 3 * j + 2);
  const C fm = s[j0 - 1], f0 = s[j0], fp = s[j0 + 1];
  return mk<C>(d1 * fm.x + d0 * f0.x + d3 * fp.x, d1 * fm.y + d0 * f0.y + d3 * fp.y);
}

// wavenumber w over the storage precision S; mean: the mean mode (w = 0);
// low: its place in the FP64 list, -1 outside it
template <typename S>
__device__ __forceinline__ void k_rhs_rows_body(int w, bool mean, int low, const RhsRowsLaunch& a) {
  using T = double;
  using C = cplx_t<T>;
  using CS = cplx_t<S>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Geom& g = a.g;
  const GridDev& gd = a.gd;
  const int j = threadIdx.x, nt = blockDim.x;
  const int ny = g.ny, n1 = g.ny1, NZ = g.nz, rk = a.rk;
  const bool row = j < n1;
  const size_t nw = (size_t)g.nw;
  const double kxd = mean ? 0.0 : gd.kx[w / NZ], kzd = mean ? 0.0 : gd.kz[w % NZ];
  const T kx = (T)kxd, kz = (T)kzd, k2 = (T)(kxd * kxd + kzd * kzd);
  CS* const gvel = (CS*)a.vel + (size_t)w * 3 * n1;
  CS* const gcru = (CS*)a.cru + (size_t)w * 3 * n1;
  CS* const gprs = (CS*)a.prs + (size_t)w * n1;
  const CS* const top = (const CS*)a.cbc_top;
  const CS* const bot = (const CS*)a.cbc_bot;
  // the FP64 columns, where this wavenumber has them (the mean's pressure is 0)
  const bool side = a.mcru64 != nullptr && (mean || low >= 0), side_p = side && !mean;
  double2* const vel64 = mean ? a.mvel64 : a.lvel64 + (ptrdiff_t)low * 3 * n1;
  double2* const cru64 = mean ? a.mcru64 : a.lcru64 + (ptrdiff_t)low * 3 * n1;
  double2* const prs64 = a.lprs64 + (ptrdiff_t)low * n1;
  C* const sV = reinterpret_cast<C*>(smem_raw);   // 3 columns of nt rows
  C* const sP = sV + 3 * nt;                      // 1 column
  const C zero = czero<C>();
  pdl_trigger();
  pdl_wait();

  // this row of cru, the nonlinear term and the pressure
  C cr[3], nl[3], p = zero;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    cr[q] = !row ? zero : side ? cru64[q * n1 + j] : cvt<C>(gcru[q * n1 + j]);
    nl[q] = row ? cvt<C>(gvel[q * n1 + j]) : zero;
  }
  if (row && !mean) p = side_p ? prs64[j] : cvt<C>(gprs[j]);
  const double dt = a.sc->dt;
  const T coef = (T)(a.rkt.B(rk) * dt);
  const T vis_imp = (T)(a.rkt.D(rk) * (dt / a.re));
  const T rk_press = (T)((a.rkt.Cc(rk) + a.rkt.D(rk)) * dt);
  const T alpha = (T)1 + vis_imp * k2;
  const T dn0 = j < ny ? (T)gd.dn[j] : (T)0, dnm1 = (j >= 1 && j <= ny) ? (T)gd.dn[j - 1] : (T)0;
  const bool uw_in = j >= 1 && j <= ny - 1, v_in = j >= 1 && j <= ny - 2;

  // cv = cru + coef*cu (+ explicit viscous term and old pressure gradient on rk1)
  C v[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = mk<C>(cr[q].x - coef * nl[q].x, cr[q].y - coef * nl[q].y);
  if (rk == 1) {
#pragma unroll
    for (int q = 0; q < 3; ++q) sV[q * nt + j] = cr[q];
    sP[j] = p;
    __syncthreads();
    const T vis_exp = (T)(a.rkt.Cc(rk) * (dt / a.re));
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int nq = q == 1 ? ny : n1;
      if (j < nq) {
        const C du = d2_of_row<T>(sV + q * nt, q == 1 ? gd.d2n : gd.d2h, j, nq);
        v[q] = cadd(v[q], cscale(vis_exp, csub(du, cscale(k2, cr[q]))));
      }
    }
    if (uw_in) {
      v[0] = csub(v[0], cimul<C>(rk_press * kx, p));
      v[2] = csub(v[2], cimul<C>(rk_press * kz, p));
    }
    if (v_in) v[1] = csub(v[1], cscale(rk_press * dn0, csub(sP[j + 1], p)));
    __syncthreads();
  }
  // the mean's constant-mass-flux pressure gradient (cu = -NL)
  double pg = 0.0;
  if (mean) {
    pg = a.sc->p_grad;
    if (a.fix_mass == 1) {
      double part = uw_in ? gd.dyh[j] * (-nl[0].x) : 0.0;
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      double* const red = reinterpret_cast<double*>(smem_raw);
      if ((j & 31) == 0) red[j >> 5] = part;
      __syncthreads();
      part = 0.0;
      for (int i = 0; i < nt >> 5; ++i) part += red[i];
      __syncthreads();
      pg = -part + 0.5 * (a.d_um_dy[ny - 1] - a.d_um_dy[0]) / a.re;
    }
    v[0].x -= (T)(cos(a.beta) * rk_press * pg);
    v[2].x -= (T)(sin(a.beta) * rk_press * pg);
  }
  // Helmholtz solves: u and w (d2h), v (d2n), wall rows from cbc or, v of the
  // FP64 list with the wall jet, in FP64
  {
    // The mean solves for its increment: with w the right-hand side and the wall
    // values, (1 - vis D2) (u - w) = vis D2 w.  The column is of size 1 and
    // nearly the same in every solve, so that a solve for u itself rounds it
    // the same way each time: 3.1e-14 off after 150 steps at 194 rows (1.8e-14
    // by elimination), 2.9e-15 with the increment.
    if (mean) {
      if (j == 0) v[0] = cvt<C>(bot[w]), v[2] = cvt<C>(bot[2 * nw + w]);
      if (j == n1 - 1) v[0] = cvt<C>(top[w]), v[2] = cvt<C>(top[2 * nw + w]);
      sV[j] = v[0];
      sV[2 * nt + j] = v[2];
      __syncthreads();
    }
    const double2* const jet = low >= 0 ? a.jet64 : nullptr;
    T ca[2] = {0, 0}, cc[2] = {0, 0}, ce[2] = {1, 1};
    C f[3] = {zero, zero, zero};
    if (j == 0) {
      if (!mean) f[0] = cvt<C>(bot[w]), f[1] = cvt<C>(bot[2 * nw + w]);
      f[2] = jet ? jet[low] : cvt<C>(bot[nw + w]);
    } else {
      if (j == n1 - 1) {
        if (!mean) f[0] = cvt<C>(top[w]), f[1] = cvt<C>(top[2 * nw + w]);
      } else if (row) {
        const T r = rcpv<T>(alpha - vis_imp * (T)gd.d2h[3 * j + 1]);
        ca[0] = vis_imp * (T)gd.d2h[3 * j] * r;
        cc[0] = vis_imp * (T)gd.d2h[3 * j + 2] * r;
        ce[0] = (T)1 - ca[0] - cc[0];
        f[0] = mean ? cscale(vis_imp * r, d2_of_row<T>(sV, gd.d2h, j, n1)) : cscale(r, v[0]);
        f[1] = mean ? cscale(vis_imp * r, d2_of_row<T>(sV + 2 * nt, gd.d2h, j, n1)) : cscale(r, v[2]);
      }
      if (j == ny - 1) {
        f[2] = jet ? jet[a.nlist + low] : cvt<C>(top[nw + w]);
      } else if (j < ny - 1) {
        const T r = rcpv<T>(alpha - vis_imp * (T)gd.d2n[3 * j + 1]);
        ca[1] = vis_imp * (T)gd.d2n[3 * j] * r;
        cc[1] = vis_imp * (T)gd.d2n[3 * j + 2] * r;
        ce[1] = (T)1 - ca[1] - cc[1];
        f[2] = cscale(r, v[1]);
      }
    }
    if (mean) __syncthreads();
    pcr_rows<T, 2, 3>(ca, cc, ce, f, n1, smem_raw);
    v[0] = mean ? cadd(v[0], f[0]) : f[0];
    v[1] = f[2];
    v[2] = mean ? cadd(v[2], f[1]) : f[1];
    if (mean) v[1] = j < ny ? cvt<C>(bot[nw]) : zero;   // the wall value
  }
  C pn = zero;
  if (!mean) {
    // strip_divergence (PFC/solve.f90:14-50) and SOLVE_P
    sV[nt + j] = v[1];
    __syncthreads();
    T ca[1] = {0}, cc[1] = {0}, ce[1] = {1};
    C f[1] = {zero};
    if (j == 0) {
      cc[0] = (T)1;
      ce[0] = (T)0;
    } else if (j == n1 - 1) {
      ca[0] = (T)1;
      ce[0] = (T)0;
    } else if (row) {
      const T dh = (T)gd.dh[j];
      const T r = rcpv<T>(dh * dnm1 + dh * dn0 + k2);
      ca[0] = dh * dnm1 * r;
      cc[0] = dh * dn0 * r;
      ce[0] = k2 * r;
      const C dv = cscale(dh, csub(v[1], sV[nt + j - 1]));
      const C s = cadd(cadd(cimul<C>(kx, v[0]), dv), cimul<C>(kz, v[2]));
      f[0] = cscale(-r / rk_press, s);
    }
    __syncthreads();
    pcr_rows<T, 1, 1>(ca, cc, ce, f, n1, smem_raw);
    sP[j] = f[0];
    __syncthreads();
    // the end rows from the one-sided wall derivative
    C ch = f[0];
    if (j == 0 || j == ny) {
      const double* dm = gd.dm + (j == 0 ? 0 : 3);
      const C p1 = sP[j == 0 ? 1 : ny - 2], p2 = sP[j == 0 ? 2 : ny - 1];
      const T m1 = (T)dm[j == 0 ? 1 : 0], m2 = (T)dm[j == 0 ? 2 : 1], m0 = (T)dm[j == 0 ? 0 : 2];
      ch = mk<C>((-m1 * p1.x - m2 * p2.x) / m0, (-m1 * p1.y - m2 * p2.y) / m0);
    }
    __syncthreads();
    if (j == 0 || j == ny) sP[j] = ch;
    __syncthreads();
    // subtract the correction gradient; p += alpha*ch - vis_imp*D2h(ch)
    if (uw_in) {
      v[0] = csub(v[0], cimul<C>(rk_press * kx, ch));
      v[2] = csub(v[2], cimul<C>(rk_press * kz, ch));
      if (v_in) v[1] = csub(v[1], cscale(rk_press * dn0, csub(sP[j + 1], ch)));
    }
    if (row) {
      const C d = d2_of_row<T>(sP, gd.d2h, j, n1);
      pn = mk<C>(p.x + alpha * ch.x - vis_imp * d.x, p.y + alpha * ch.y - vis_imp * d.y);
    }
    __syncthreads();
  }
  // next-substep accumulator (PFC/pass2.f90:312-333)
#pragma unroll
  for (int q = 0; q < 3; ++q) sV[q * nt + j] = v[q];
  sP[j] = pn;
  __syncthreads();
  C acc[3] = {v[0], v[1], v[2]};
  if (rk < 3) {
    const T coef2 = (T)(dt * a.rkt.A(rk + 1));
    const T vis_exp2 = (T)((dt / a.re) * a.rkt.Cc(rk + 1));
    const T rkp2 = (T)((a.rkt.Cc(rk + 1) + a.rkt.D(rk + 1)) * dt);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int nq = q == 1 ? ny : n1;
      acc[q] = mk<C>(v[q].x - coef2 * nl[q].x, v[q].y - coef2 * nl[q].y);
      if (j < nq) {
        const C du = d2_of_row<T>(sV + q * nt, q == 1 ? gd.d2n : gd.d2h, j, nq);
        acc[q] = cadd(acc[q], cscale(vis_exp2, csub(du, cscale(k2, v[q]))));
      }
    }
    if (uw_in) {
      acc[0] = csub(acc[0], cimul<C>(rkp2 * kx, pn));
      acc[2] = csub(acc[2], cimul<C>(rkp2 * kz, pn));
    }
    if (v_in) acc[1] = csub(acc[1], cscale(rkp2 * dn0, csub(sP[j + 1], pn)));
  }
  if (row) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      gvel[q * n1 + j] = cvt<CS>(v[q]);
      gcru[q * n1 + j] = cvt<CS>(acc[q]);
      if (side) {
        vel64[q * n1 + j] = v[q];
        cru64[q * n1 + j] = acc[q];
      }
    }
    gprs[j] = cvt<CS>(pn);
    if (side_p) prs64[j] = pn;
  }
  if (mean) {
    const double* dm = gd.dm;
    if (j == 0) {
      a.sc->p_grad = pg;
      if (a.advance) a.sc->t_total = a.sc->t_total + dt;
      a.d_um_dy[0] = dm[0] * sV[0].x + dm[1] * sV[1].x + dm[2] * sV[2].x;
      a.d_um_dy[ny - 1] = dm[3] * sV[ny - 2].x + dm[4] * sV[ny - 1].x + dm[5] * sV[ny].x;
    }
    if (v_in) a.d_um_dy[j] = dn0 * (sV[j + 1].x - v[0].x);
  }
}

// block b of the launch: the mean mode (a.mean), the FP64 list, the fast list
template <typename S>
__device__ __forceinline__ void k_rhs_rows_block(int b, const RhsRowsLaunch& a) {
  const int i = b - a.mean;   // place in the FP64 list, then in the fast list
  k_rhs_rows_body<S>(i < 0 ? 0 : i < a.nlist ? a.wlist[i] : a.wfast[i - a.nlist], i < 0, i < a.nlist ? i : -1, a);
}

}  // namespace cfd
