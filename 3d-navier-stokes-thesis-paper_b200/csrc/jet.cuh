// jet.cuh -- crossflow wall forcing cbc(:,:,2) on the device: jet_profile
// (PFC/pass2.f90:423-673) for a closed channel (bl_grid = 0).
//   k_jet_walk    : end-of-substep time and the random walk of the Freund
//                   forcing parameters (:454-477), RANDOM_NUMBER replaced by
//                   the counter RNG: draw n of call k is u01(seed, k, 0, n, 7)
//   k_jet_field   : physical planes on the nx x nz grid: the suction profile
//                   (define_suction_profile, :553-609) and the jet outflow of
//                   each forced wall (define_jet_profile, :611-656, or the
//                   Gaussian spanwise slot)
//   k_jet_combine : after the small forward transforms: filter_cosine passes
//                   (:658-671), top-wall sign, suction balance (:493-537)
//   k_jet_low     : mixed precision: the same coefficients in FP64 for the
//                   |k| < 4 list
#pragma once
#include <cstdint>

#include "cfd_common.cuh"
#include "pass1.cuh"
#include "pass2.cuh"

namespace cfd {

struct JetParams {
  int mode;                        // 0 off, 1 tanh jet, 2 Gaussian slot
  double xjet[2], zjet[2], jetmag[2], forcing[2], for_freq[2];
  double jet_diam, width, freq, frac_xbuff;
  int filter;
  unsigned long long seed;
};

struct JetState {
  double jf[24], inc[24];   // (3,2,4) parameters and increments
  double time, incr;        // of the current call
  long long calls;
};

__device__ __forceinline__ uint64_t jet_smix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}
// the counter RNG shared with the host initial-field generator
__device__ __forceinline__ double jet_u01(uint64_t seed, long long x, int z, int j, int col) {
  const uint64_t ctr = ((((uint64_t)x * 65536u + (uint64_t)z) * 65536u + (uint64_t)j) * 8u) + (uint64_t)col;
  const uint64_t h = jet_smix(seed ^ jet_smix(ctr));
  return (double)(h >> 11) * (1.0 / 9007199254740992.0);
}

// one warp.  use_sc: time = t_total + dt*sum(rkc(1:rk)+rkd(1:rk)),
// incr = dt*(rkc(rk)+rkd(rk)) from the device scalars (PFC/pass2.f90:37-38);
// otherwise the given time/incr.
__device__ __forceinline__ void k_jet_walk_body(const uint3 bid, JetState* __restrict__ st, JetParams jp,
                                                const DevScalars* __restrict__ sc, RkTab rkt, int rk, double time,
                                                double incr, int use_sc) {
  const int n = threadIdx.x;
  if (use_sc) {
    double s = 0.0;
    for (int r = 1; r <= rk; ++r) s += rkt.Cc(r) + rkt.D(r);
    time = sc->t_total + sc->dt * s;
    incr = sc->dt * (rkt.Cc(rk) + rkt.D(rk));
  }
  const long long k = st->calls;
  __syncwarp();
  if (n == 0) { st->time = time; st->incr = incr; st->calls = k + 1; }
  if (jp.seed == 0 || n >= 24) return;
  const double r = jet_u01(jp.seed, k, 0, n, 7);
  double inc = st->inc[n] * ((r - 0.05) >= 0.0 ? 1.0 : -1.0);   // SIGN(1, r - 0.05)
  double f = st->jf[n] + incr * inc;
  const int kk = n / 6;   // (i,j,k): n = i + 3 j + 6 k
  if (kk == 0) {
    if (f <= 0.01) { f = 0.01; inc = fabs(inc); }
    else if (f >= 0.07) { f = 0.07; inc = -fabs(inc); }
  } else if (kk == 1) {
    if (f <= 0.1) { f = 0.1; inc = fabs(inc); }
    else if (f >= 0.7) { f = 0.7; inc = -fabs(inc); }
  }
  st->jf[n] = f;
  st->inc[n] = inc;
}

__global__ void k_jet_walk(JetState* __restrict__ st, JetParams jp, const DevScalars* __restrict__ sc, RkTab rkt,
                           int rk, double time, double incr, int use_sc) {
  k_jet_walk_body(blockIdx, st, jp, sc, rkt, rk, time, incr, use_sc);
}

// |(a, b)| of a default-real complex: both parts rounded to single, the
// modulus formed in double and rounded to single
__device__ __forceinline__ double abs_cmplx_single(double a, double b) {
  const double af = (double)(float)a, bf = (double)(float)b;
  return (double)(float)sqrt(af * af + bf * bf);
}

// grid (nz, 3), block 128: planes 0 suction, 1 bottom jet, 2 top jet;
// phys[p][z][x] on the nx x nz grid.  With rows64: also the row's first nk
// coefficients in FP64, rows64[p][kx][z] (not scaled), by direct sums;
// dynamic shared memory jet_row_smem(nx)
__host__ __device__ __forceinline__ size_t jet_row_smem(int nx) { return (size_t)nx * (sizeof(double2) + sizeof(double)); }
template <typename T>
__device__ __forceinline__ void k_jet_field_body(const uint3 bid, T* __restrict__ phys, double2* __restrict__ rows64,
                                                 int nk, JetParams jp,
                                                 const JetState* __restrict__ st, int nx, int nz, double lx,
                                                 double lz) {
  const int z = bid.x, p = bid.y;
  const double pi = 3.14159265358979323846;
  const double time = st->time;
  const double zc = (double)z * lz / (double)nz;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* const tw = reinterpret_cast<double2*>(smem_raw);   // exp(-2 pi i m / nx)
  double* const row = reinterpret_cast<double*>(tw + nx);
  for (int x = threadIdx.x; x < nx; x += blockDim.x) {
    const double xc = (double)x * lx / (double)nx;
    double v = 0.0;
    if (p == 0) {
      const double frac_suct = 0.5 * jp.frac_xbuff, suct_start = 1.0 - jp.frac_xbuff;
      const double suct_rise = 0.25 * frac_suct, suct_fall = 0.25 * frac_suct;
      const double xstart = lx * suct_start, xrise = xstart + lx * suct_rise;
      const double xfall = xstart + lx * frac_suct - lx * suct_fall, xend = xstart + lx * frac_suct;
      if (xc > xstart && xc < xend) {
        if (xc < xrise) {
          const double x2 = (xc - xstart) / (xrise - xstart);
          v = 1.0 / (1.0 + exp(1.0 / x2 + 1.0 / (x2 - 1.0)));
        } else if (xc > xfall) {
          const double x2 = (xend - xc) / (xend - xfall);
          v = 1.0 / (1.0 + exp(1.0 / x2 + 1.0 / (x2 - 1.0)));
        } else {
          v = 1.0;
        }
      }
    } else {
      const int w = p - 1;
      const double jm = jp.jetmag[w];
      if (jp.mode == 1 && jm != 0.0) {
        const double v_ampl = jm * (1.0 + jp.forcing[w] * sin(2.0 * pi * time * jp.for_freq[w] * jm / jp.jet_diam));
        const double xd1 = xc - jp.xjet[w], xd2 = xc - (lx + jp.xjet[w]);
        const double zd1 = zc - jp.zjet[w], zd2 = zc - (lz + jp.zjet[w]);
        const double r1 = abs_cmplx_single(xd1, zd1) * 2.0 / jp.jet_diam;
        const double r2 = abs_cmplx_single(xd2, zd1) * 2.0 / jp.jet_diam;
        const double r3 = abs_cmplx_single(xd1, zd2) * 2.0 / jp.jet_diam;
        const double r4 = abs_cmplx_single(xd2, zd2) * 2.0 / jp.jet_diam;
        const double r = fmin(fmin(r1, r2), fmin(r3, r4));
        if (r == 0.0) {
          v = v_ampl;
        } else {
          const double phi = atan2(zd1, xd1);
          double s = 0.0;
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            const double fw = (double)(i % 3);
            s += st->jf[i] * cos(st->jf[6 + i] * jm * time / jp.jet_diam + st->jf[12 + i]) *
                 cos(fw * phi + st->jf[18 + i]);
          }
          const double bjet = 5.0 + s;
          v = v_ampl * 0.5 * (1.0 - tanh(bjet * (r - 1.0 / r)));
        }
      } else if (jp.mode == 2 && jm != 0.0) {
        const double a = jm * 0.5 * (1.0 + sin(2.0 * pi * jp.freq * time));
        double d = fabs(xc - jp.xjet[w]);
        if (lx - d < d) d = lx - d;
        v = a * exp(-(d / jp.width) * (d / jp.width));
      }
    }
    phys[((size_t)p * nz + z) * nx + x] = (T)v;
    if (rows64) {
      row[x] = v;
      sincospi(-2.0 * (double)x / (double)nx, &tw[x].y, &tw[x].x);
    }
  }
  if (!rows64) return;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int kx = threadIdx.x >> 5; kx < nk; kx += blockDim.x >> 5) {
    double re = 0.0, im = 0.0;
    for (int x = lane; x < nx; x += 32) {
      const double2 c = tw[kx * x % nx];
      re += row[x] * c.x;
      im += row[x] * c.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (lane == 0) rows64[((size_t)p * nk + kx) * nz + z] = make_double2(re, im);
  }
}

template <typename T>
__global__ void k_jet_field(T* __restrict__ phys, double2* __restrict__ rows64, int nk, JetParams jp,
                            const JetState* __restrict__ st, int nx, int nz, double lx, double lz) {
  k_jet_field_body<T>(blockIdx, phys, rows64, nk, jp, st, nx, nz, lx, lz);
}

// spec[p][kx][kz] (p = 0 suction, 1 bottom, 2 top) -> cbc(:,:,2) of the
// forced walls, the other wall slots zeroed
template <typename T>
__device__ __forceinline__ void k_jet_combine_body(const uint3 bid, const cplx_t<T>* __restrict__ spec,
                                                   cplx_t<T>* __restrict__ cbc, JetParams jp, GridDev gd, int nx,
                                                   int nz, int nxh, double lx, double lz) {
  using C = cplx_t<T>;
  const int nw = nz * nxh;
  const int w = bid.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  const int kx = w / nz, kz = w % nz;
  const double pi = 3.14159265358979323846;
  const double fx = 1.0 + cos(pi * gd.kx[kx] / ((double)(nx / 2) * 2.0 * pi / lx));
  const double fz = 1.0 + cos(pi * gd.kz[kz] / ((double)(nz / 2) * 2.0 * pi / lz));
  auto filt = [&](C v) {
    double re = (double)v.x, im = (double)v.y;
    for (int n = 0; n < jp.filter; ++n) {
      re = re * 0.5 * fx * 0.5 * fz;
      im = im * 0.5 * fx * 0.5 * fz;
    }
    return mk<C>((T)re, (T)im);
  };
  // the (0,0) coefficients carry the filter factor 1
  const C cs = filt(spec[w]);
  const double sum_suction = (double)spec[0].x;
  for (int wall = 0; wall < 2; ++wall) {
    C out = czero<C>();
    if (jp.mode != 0 && jp.jetmag[wall] != 0.0) {
      const double sg = wall == 1 ? -1.0 : 1.0;
      const C cj = filt(spec[(size_t)(1 + wall) * nw + w]);
      const double sum = sg * (double)spec[(size_t)(1 + wall) * nw].x;
      const double q = sum / sum_suction;
      out = mk<C>((T)(sg * (double)cj.x - q * (double)cs.x), (T)(sg * (double)cj.y - q * (double)cs.y));
    }
    // cbc layout [bot, top][comp][kx][kz]: component 2 (v) is index 1
    cbc[((size_t)wall * 3 + 1) * nw + w] = out;
  }
}

template <typename T>
__global__ void k_jet_combine(const cplx_t<T>* __restrict__ spec, cplx_t<T>* __restrict__ cbc, JetParams jp,
                              GridDev gd, int nx, int nz, int nxh, double lx, double lz) {
  k_jet_combine_body<T>(blockIdx, spec, cbc, jp, gd, nx, nz, nxh, lx, lz);
}

// k_jet_low: grid (n), block 128: the forced walls' coefficients of the list's
// wavenumbers in FP64, out[wall][n], by direct sums over z of the rows'
// coefficients rows64.  The change of a wall value from substep to substep
// reaches the pressure divided by k dt, and the rounding of FP32 values with
// it: 1e-6 of velocity and pressure together, all of it in the lowest few kx
// (36x46x24, dt 0.002, jet amplitude 0.1).  Nyquist coefficients keep the FP32
// value (cbc, after k_jet_combine).  Sums over the whole planes instead took
// 75 us a substep at 128x129x128, more than the jet has beside the nonlinear
// term.
__device__ __forceinline__ void k_jet_low_body(int i, int n, const int* __restrict__ list,
                                               const double2* __restrict__ rows64, int nk,
                                               const float2* __restrict__ cbc, double2* __restrict__ out, JetParams jp,
                                               GridDev gd, int nx, int nz, int nxh, double lx, double lz) {
  __shared__ double red[9][4];
  const int w = list[i], kx = w / nz, kz = w % nz, t = threadIdx.x;
  const size_t np = (size_t)nx * nz, nw = (size_t)nz * nxh;
  double a[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};   // per plane: the coefficient, the mean
  for (int z = t; z < nz; z += 128) {
    double sn, cs;
    sincospi(-2.0 * (double)((long long)kz * z % nz) / (double)nz, &sn, &cs);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const double2 v = rows64[((size_t)p * nk + kx) * nz + z];
      a[3 * p] += v.x * cs - v.y * sn;
      a[3 * p + 1] += v.x * sn + v.y * cs;
      a[3 * p + 2] += rows64[(size_t)p * nk * nz + z].x;
    }
  }
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    for (int o = 16; o > 0; o >>= 1) a[r] += __shfl_xor_sync(0xffffffffu, a[r], o);
    if ((t & 31) == 0) red[r][t >> 5] = a[r];
  }
  __syncthreads();
  if (t >= 2) return;
#pragma unroll
  for (int r = 0; r < 9; ++r) a[r] = red[r][0] + red[r][1] + red[r][2] + red[r][3];
  const int wall = t;
  if (kx == nx / 2 || kz == nz / 2) {
    const float2 v = cbc[((size_t)wall * 3 + 1) * nw + w];
    out[(size_t)wall * n + i] = make_double2((double)v.x, (double)v.y);
    return;
  }
  double2 v = make_double2(0.0, 0.0);
  if (jp.mode != 0 && jp.jetmag[wall] != 0.0) {
    const double pi = 3.14159265358979323846;
    const double fx = 1.0 + cos(pi * gd.kx[kx] / ((double)(nx / 2) * 2.0 * pi / lx));
    const double fz = 1.0 + cos(pi * gd.kz[kz] / ((double)(nz / 2) * 2.0 * pi / lz));
    double f = 1.0 / (double)np;
    for (int r = 0; r < jp.filter; ++r) f *= 0.25 * fx * fz;
    const double sg = wall == 1 ? -1.0 : 1.0;
    const double q = sg * (wall ? a[8] : a[5]) / a[2];
    v = make_double2(f * (sg * (wall ? a[6] : a[3]) - q * a[0]), f * (sg * (wall ? a[7] : a[4]) - q * a[1]));
  }
  out[(size_t)wall * n + i] = v;
}

__global__ void __launch_bounds__(128) k_jet_low(int n, const int* __restrict__ list,
                                                 const double2* __restrict__ rows64, int nk,
                                                 const float2* __restrict__ cbc, double2* __restrict__ out,
                                                 JetParams jp, GridDev gd, int nx, int nz, int nxh, double lx,
                                                 double lz) {
  k_jet_low_body((int)blockIdx.x, n, list, rows64, nk, cbc, out, jp, gd, nx, nz, nxh, lx, lz);
}

// ---------------------------------------------------------------------------
// init_buffer (PFC/init_jet_buffer.f90:358-483): the fringe profile on the
// nx x nz grid.  Each direction's band rises and falls with
// 1/(1+exp(1/t + 1/(t-1))) (define_fringe_region, :453-482); where the x and
// z bands overlap the two ramps combine through sqrt(tx^2 + tz^2).
struct FringeParams {
  int xfringe, zfringe;
  double frac_xbuff, buff_xrise, buff_xfall, frac_zbuff;
};

__device__ __forceinline__ void fringe_region(double t, double ts, double tr, double tf, double te, double& f,
                                              double& f2) {
  f = 0.0;
  f2 = 0.0;
  if (t > ts) {
    if (t < tr) {
      const double t2 = (t - ts) / (tr - ts);
      f = 1.0 / (1.0 + exp(1.0 / t2 + 1.0 / (t2 - 1.0)));
      f2 = t2;
    } else if (t > tf && t < te) {
      const double t2 = (te - t) / (te - tf);
      f = 1.0 / (1.0 + exp(1.0 / t2 + 1.0 / (t2 - 1.0)));
      f2 = t2;
    } else if (t >= te) {
      f = 0.0;
    } else {
      f = 1.0;
    }
  }
}

template <typename T>
__global__ void k_fringe_profile(T* __restrict__ out, FringeParams fp, int nx, int nz, double lx, double lz) {
  const int z = blockIdx.x;
  const double tz = (double)z * lz / (double)nz;
  double fz = 0.0, fz2 = 0.0;
  if (fp.zfringe == 1) {
    double fa, fa2, fb, fb2;
    fringe_region(tz, -1.0, -1.0, 0.0, fp.frac_zbuff * lz, fa, fa2);
    fringe_region(tz, lz - fp.frac_zbuff * lz, lz, lz + 1.0, lz + 1.0, fb, fb2);
    fz = fa + fb;
    fz2 = fa2 + fb2;
  }
  for (int x = threadIdx.x; x < nx; x += blockDim.x) {
    const double tx = (double)x * lx / (double)nx;
    double fx = 0.0, fx2 = 0.0;
    if (fp.xfringe == 1) {
      const double xs = lx * (1.0 - fp.frac_xbuff);
      fringe_region(tx, xs, xs + lx * fp.buff_xrise, lx - lx * fp.buff_xfall, lx, fx, fx2);
    }
    double v;
    if (fx < 1.0 && fz < 1.0 && fx * fz > 0.0) {
      const double t = sqrt(fx2 * fx2 + fz2 * fz2);
      v = (t < 1.0) ? 1.0 / (1.0 + exp(1.0 / t + 1.0 / (t - 1.0))) : 1.0;
    } else {
      v = fmax(fx, fz);
    }
    out[(size_t)z * nx + x] = (T)v;
  }
}

template <typename T>
__global__ void k_scale_real(const T* __restrict__ in, T* __restrict__ out, size_t n, double s) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = (T)(s * (double)in[i]);
}

}  // namespace cfd
