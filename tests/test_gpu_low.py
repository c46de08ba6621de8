"""Mixed precision: the FP64 columns of the |k| < 4 wavenumbers.

- The error of a run.  A rounding of these columns reaches the pressure
  divided by k^2 dt, so their FP32 rounding set the error of velocity and
  pressure together: 2e-7 to 3e-7 of their norm on the first five of these
  grids, beyond 1e-6 with larger disturbances.  With the columns in FP64 what
  is left is the rounding of the FP32 transforms, 1.2e-7 of the nonlinear term
  at every length, and of the |k| >= 4 columns, whose part of the pressure is
  at least 16 times smaller: the bar, against the same run in FP64, is 1.2e-7.
- The wall jet, whose rounding in FP32 changes from substep to substep and
  reaches the pressure divided by k dt: 1e-6 of the norm, all of it at kx of
  0.5 and 1.  Its coefficients at |k| < 4 are in FP64; the others' part is at
  most an eighth of that.  The bar: an eighth of 1e-6 and the 1.2e-7 of a run.
- Where the columns can go out of date or get lost: a state taken out and put
  back (at the end of a step and within one, through the arrays and through
  the restart file), the learned closure's solves, which read the FP32
  columns, and the autotuner's trial steps.  The run goes on bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LX, LZ = 4 * np.pi, 2 * np.pi


def flow_of(cf, nx, ny, nz, prec, dt=0.004):
    return cf.ChannelFlow(cf.Grid(nx, ny, nz, lx=LX, lz=LZ, stretch=1.5), re=2500.0, dt=dt, precision=prec)


def field(f, seed):
    """The laminar profile and noise that falls off as k^-2, smooth in y, as FP32 holds them."""
    rng = np.random.default_rng(seed)
    nz, nxh, n1, _ = f.shapes()[0]
    g = f.grid
    kx, kz = np.asarray(g.kx).ravel()[None, :], np.asarray(g.kz).ravel()[:, None]
    c = rng.standard_normal((2, nz, nxh, 3)) + 1j * rng.standard_normal((2, nz, nxh, 3))
    c *= 1e-2 * np.minimum(1.0, 1.0 / np.maximum(kx ** 2 + kz ** 2, 1e-30))[None, :, :, None]
    c[:, nz // 2] = 0
    c[:, :, nxh - 1] = 0
    c[:, nz // 2 + 1:, 0] = np.conj(c[:, 1:nz // 2, 0][:, ::-1])
    c[:, 0, 0] = 0
    d1 = np.zeros(f.shapes()[0], np.complex128, order="F")
    yh = np.asarray(g.yh).ravel()
    y = np.append(np.asarray(g.y).ravel(), 1.0)
    for q, yy in ((0, yh), (1, y), (2, yh)):
        p = np.stack([1 - yy ** 2, yy]) * (1 - yy ** 2)
        d1[..., q] = np.einsum("mj,mzx->zxj", p, c[..., q])
    d1 = np.asfortranarray(d1.astype(np.complex64).astype(np.complex128))
    d1[0, 0, :, 0] = 1 - yh ** 2
    return d1


def start(f, seed):
    f.upload_state(field(f, seed), None, np.zeros(f.shapes()[2], np.complex128, order="F"))
    f.remove_initial_divergence()
    f.compute_initial_pressure(0)


def state(f):
    s = f.scalars()
    return f.download_state(), (s["t_total"], s["dt"], s["p_grad"], s["d_um_dy"])


def restore(f, s):
    f.upload_state(*s[0])
    f.set_scalars(*s[1])


def same(a, b):
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(a[1][3], b[1][3])
    assert a[1][:3] == b[1][:3]


@pytest.mark.parametrize("nx,ny,nz,dt", [(32, 55, 144, 0.002), (32, 20, 216, 0.002), (16, 40, 32, 0.002),
                                         (72, 45, 16, 0.0025), (36, 31, 32, 0.004), (64, 130, 32, 0.004)])
def test_error_of_a_run(cf, nx, ny, nz, dt):
    out = []
    for prec in (0, 1):
        f = flow_of(cf, nx, ny, nz, prec, dt)
        start(f, nx)
        f.timestep(40)
        d1, _, d4 = f.download_state()
        assert f.status() == 0
        out.append(np.concatenate([d1.ravel(), d4.ravel()]))
        f.close()
    err = np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0])
    assert err < 1.2e-7, err


def slot_jet(cf):
    j = cf.CfgJet()
    j.mode = 2
    j.xjet[0], j.zjet[0] = 0.3 * LX, 0.5 * LZ
    j.jetmag[0] = 0.1
    j.width, j.freq, j.frac_xbuff, j.seed = 0.2, 0.5, 0.2, 2
    return j


@pytest.mark.parametrize("dt_flag", [0, 1])
@pytest.mark.parametrize("nx,ny,nz,dt", [(36, 46, 24, 0.002), (32, 86, 36, 0.002), (96, 30, 48, 0.002)])
def test_error_of_a_run_with_the_wall_jet(cf, nx, ny, nz, dt, dt_flag):
    out = []
    for prec in (0, 1):
        f = cf.ChannelFlow(cf.Grid(nx, ny, nz, lx=LX, lz=LZ, stretch=1.5), re=3000.0, dt=dt, precision=prec,
                           dt_flag=dt_flag, cfl_max=0.05)
        start(f, nx)
        f.set_jet(slot_jet(cf))
        f.timestep(40)
        d1, _, d4 = f.download_state()
        assert f.status() == 0
        out.append(np.concatenate([d1.ravel(), d4.ravel()]))
        f.close()
    err = np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0])
    assert err < 2.45e-7, err


@pytest.mark.parametrize("nx,ny,nz", [(32, 33, 32), (96, 40, 96)])
def test_state_out_and_back(cf, tmp_path, nx, ny, nz):
    a, b = flow_of(cf, nx, ny, nz, 1), flow_of(cf, nx, ny, nz, 1)
    start(a, 3)
    a.timestep(3)
    restore(b, state(a))
    same(state(b), state(a))
    for f in (a, b):
        f.timestep(3)
    same(state(b), state(a))
    a.nonlinear(7, 1)
    a.rhs_solve(7, 1)
    restore(b, state(a))
    for f in (a, b):
        f.nonlinear(7, 2)
        f.rhs_solve(7, 2)
    same(state(b), state(a))
    path = str(tmp_path / "v.out")
    a.save_velocity(path, wait=True)
    start(b, 4)
    b.timestep(1)
    b.read_velocity(path)
    np.testing.assert_array_equal(b.download_state()[0], a.download_state()[0])


def test_learned_closure_and_back(cf):
    """The learned closure's steps leave their FP32 columns to what follows."""
    rng = np.random.default_rng(5)
    net = cf.Mlp(params=(0.1 * rng.standard_normal(9414)).astype(np.float32))
    a, b = flow_of(cf, 32, 33, 32, 1), flow_of(cf, 32, 33, 32, 1)
    start(a, 6)
    for model in (0, 1):
        a.timestep(2)
        a.set_les(2, mlp=net)
        a.timestep(2)
        kept = state(a)
        a.set_les(model)
        same(state(a), kept)
        b.set_les(model)
        restore(b, kept)
        for f in (a, b):
            f.timestep(3)
        same(state(b), state(a))


def test_autotune_restores(cf):
    a, b = flow_of(cf, 48, 33, 48, 1), flow_of(cf, 48, 33, 48, 1)
    for f in (a, b):
        start(f, 8)
        f.timestep(2)
    a.autotune(2)
    same(state(a), state(b))
    for f in (a, b):
        f.timestep(2)
    same(state(a), state(b))


@pytest.mark.parametrize("batched", [True, False])
def test_ensemble_graph_after_learned_steps(cf, batched):
    """A captured ensemble step goes on from what its members did by themselves in between."""
    rng = np.random.default_rng(5)
    net = cf.Mlp(params=(0.1 * rng.standard_normal(9414)).astype(np.float32))
    m = [flow_of(cf, 32, 33, 32, 1) for _ in range(2)]
    alone = flow_of(cf, 32, 33, 32, 1)
    for i, f in enumerate(m):
        start(f, 20 + i)
    ens = cf.Ensemble(m, autotune=False, batched=batched)
    ens.timestep(4)
    ens.synchronize()
    m[1].set_les(2, mlp=net)
    m[1].timestep(2)
    restore(alone, state(m[1]))
    ens.timestep(3)
    ens.synchronize()
    alone.timestep(3)
    same(state(m[1]), state(alone))
    ens.close()


def test_steps_after_a_captured_learned_member(cf):
    rng = np.random.default_rng(6)
    net = cf.Mlp(params=(0.1 * rng.standard_normal(9414)).astype(np.float32))
    m = [flow_of(cf, 32, 33, 32, 1) for _ in range(2)]
    alone = flow_of(cf, 32, 33, 32, 1)
    for i, f in enumerate(m):
        start(f, 30 + i)
    m[1].set_les(2, mlp=net)
    ens = cf.Ensemble(m, autotune=False)
    ens.timestep(3)
    ens.synchronize()
    m[1].set_les(0)
    ens.timestep(2)       # the captured step is the learned one
    ens.synchronize()
    restore(alone, state(m[1]))
    for f in (m[1], alone):
        f.timestep(2)
    same(state(m[1]), state(alone))
    ens.close()
