"""The mean mode over a run.  A state that is nothing but mean columns has no
nonlinear term, so that its time steps are three tridiagonal solves for u and
w each with the constant-mass-flux pressure gradient; restated here in
extended precision.  The column is nearly the same in every solve, and a
solver that rounds it the same way each time drifts from it linearly in time:
150 steps end no further from the extended-precision columns than the same
steps in FP64 with plain elimination."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RKA, RKB, RKC, RKD = ([float(np.float32(v)) for v in t] for t in (
    (0.0, -17.0 / 60.0, -5.0 / 12.0), (8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0), (29.0 / 96.0, -3.0 / 40.0, 1.0 / 6.0),
    (37.0 / 160.0, 5.0 / 24.0, 1.0 / 6.0)))


def columns(grid, u, re, dt, steps, T):
    """u: (rows, 2) columns of u and w after the steps, in precision T, by elimination."""
    d2, dm = np.asarray(grid.d2h).T.astype(T), np.asarray(grid.dm).ravel(order="F").astype(T)
    n, re, dt = len(u), T(re), T(dt)
    u = u.astype(T)
    near = np.clip(np.arange(n), 1, n - 2)

    def diff(f):
        return d2[:, :1] * f[near - 1] + d2[:, 1:2] * f[near] + d2[:, 2:] * f[near + 1]

    def shear(f):
        return dm[:3] @ f[:3, 0], dm[3:6] @ f[-3:, 0]

    cru = u.copy()
    for _ in range(steps):
        for rk in range(3):
            lo, hi = shear(u)
            vis, press = T(RKD[rk]) * (dt / re), (T(RKC[rk]) + T(RKD[rk])) * dt
            v = cru.copy()
            if rk == 0:
                v += T(RKC[0]) * (dt / re) * diff(cru)
            v[:, 0] -= press * (T(0.5) * (hi - lo) / re)
            v[0] = v[-1] = 0
            a, b, c = -vis * d2[:, 0], 1 - vis * d2[:, 1], -vis * d2[:, 2]
            a[[0, -1]], b[[0, -1]], c[[0, -1]] = 0, 1, 0
            for i in range(1, n):
                m = a[i] / b[i - 1]
                b[i] -= m * c[i - 1]
                v[i] -= m * v[i - 1]
            v[-1] /= b[-1]
            for i in range(n - 2, -1, -1):
                v[i] = (v[i] - c[i] * v[i + 1]) / b[i]
            u = v
            cru = u + (dt / re) * T(RKC[rk + 1]) * diff(u) if rk < 2 else u.copy()
    return u, shear(u)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny,re,dt", [(16, 193, 2500.0, 0.005), (16, 64, 2500.0, 0.005), (48, 129, 400.0, 0.01)])
def test_mean_columns_of_a_run(cf, nx, ny, re, dt, prec):
    grid = cf.Grid(nx, ny, nx, stretch=1.5)
    yh = np.asarray(grid.yh).ravel()
    u0 = np.stack([1 - yh ** 2, 0.1 * (1 - yh ** 2) * yh], 1)
    exact, shear = columns(grid, u0, re, dt, 150, np.longdouble)
    plain, _ = columns(grid, u0, re, dt, 150, np.float64)
    f = cf.ChannelFlow(grid, re=re, dt=dt, precision=prec)
    s1, s2, s4 = f.shapes()
    d1, d2 = np.zeros(s1, np.complex128, order="F"), np.zeros(s2, np.complex128, order="F")
    d1[0, 0, :, 0], d1[0, 0, :, 2] = u0[:, 0], u0[:, 1]
    d2[:, 0, 0, 0], d2[:, 2, 0, 0] = u0[:, 0], u0[:, 1]
    f.upload_state(d1, d2, np.zeros(s4, np.complex128, order="F"))
    dm = np.asarray(grid.dm).ravel(order="F")
    dud = np.zeros(ny)
    dud[0], dud[-1] = dm[:3] @ u0[:3, 0], dm[3:6] @ u0[-3:, 0]
    f.set_scalars(0.0, dt, 0.0, dud)
    f.timestep(150)
    assert f.status() == 0
    got = f.download_state()[0]
    other = got.copy()
    other[0, 0] = 0
    assert not other.any()
    got = got[0, 0][:, [0, 2]]
    assert not got.imag.any()

    def off(a):
        return float(np.linalg.norm(a - exact) / np.linalg.norm(exact))

    assert off(got.real) <= off(plain), (off(got.real), off(plain))
    f.close()
