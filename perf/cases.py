"""The work that users of the channel-flow framework have it do, as cases that
can be timed: direct numerical simulation from the smallest grids to the
largest, in both precisions, with fixed and adaptive time step, with wall jet
and wall feedback; large-eddy simulation with the eddy viscosity and with the
learned closure; training that closure; ensembles of small domains; and the
propagator of the stability solver.

listed() are the cases, draw(rng) gives more of the same ranges, prepare()
makes what a program holds before the call (context, state, buffers), run()
is one pass through the public entry points: a number of time steps, and the
state brought back to the host as a program does between outputs: the
velocity and the pressure, one after the other as in a snapshot file, in the
precision in which the context holds them (FP32 in mixed precision; the host
arrays of the C ABI are FP64).

exact() restates the same pass in 64 bits with torch alone: grid operators,
dealiased transforms, staggered fluxes, the RK3/Crank-Nicolson substeps with
their tridiagonal solves, wall conditions, subgrid stresses, and the network.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

cf = importlib.import_module("3d-navier-stokes-thesis-paper_b200.chanflow")

LX, LZ, STRETCH = 4 * math.pi, 2 * math.pi, 1.5
# transform lengths must be 2^a 3^b with even 3/2 multiples
LENGTHS = (16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256, 288, 384)
LARGEST = 384 * 193 * 384
ENS_GRIDS = ((48, 49, 48), (64, 65, 64), (96, 97, 96))


# ---------------------------------------------------------------- the cases
def _dns(nx, ny, nz, precision, steps, re=2500.0, dt=0.005, ampl=1e-2, adaptive=False, jet=False, feedback=False):
    return {"kind": "dns", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "steps": steps, "re": re,
            "dt": dt, "ampl": ampl, "adaptive": adaptive, "jet": jet, "feedback": feedback}


def listed():
    return [
        # a quick run of the smallest configuration (a new user's first flow.dat, a parameter sweep): launches count
        dict(_dns(32, 33, 32, "mixed", 20), name="dns_32_mixed"),
        # flow control at moderate size: Gaussian wall jet and wall-shear feedback
        dict(_dns(128, 129, 128, "mixed", 30, re=2800.0, dt=0.0025, jet=True, feedback=True), name="control_128_mixed"),
        # the grid of the reference's published run, adaptive time step
        dict(_dns(128, 200, 64, "mixed", 40, re=5000.0, adaptive=True), name="dns_128x200x64_adaptive"),
        # the headline configuration, in both precisions
        dict(_dns(256, 193, 256, "mixed", 40, ampl=1e-3), name="dns_256_mixed"),
        dict(_dns(256, 193, 256, "fp64", 15, ampl=1e-3), name="dns_256_fp64"),
        # the largest: the DNS that an LES closure is trained on
        dict(_dns(384, 193, 384, "mixed", 30, re=10350.0, dt=0.002, adaptive=True), name="dns_384_mixed"),
        # a grid off the powers of two, with an even number of planes
        dict(_dns(144, 100, 108, "mixed", 20), name="dns_144x100x108_mixed"),
        # LES on a coarse grid, eddy viscosity and learned closure
        {"name": "les_eddy_128", "kind": "les", "nx": 128, "ny": 65, "nz": 128, "model": 1, "steps": 40, "re": 10350.0},
        {"name": "les_learned_128", "kind": "les", "nx": 128, "ny": 65, "nz": 128, "model": 2, "steps": 20,
         "re": 10350.0},
        # fitting the closure network: one update from the gradients of 16 batches of the pipeline's own size
        {"name": "train_4096", "kind": "train", "batch": 4096, "samples": 1000000, "batches": 16},
        # many small domains on one GPU
        {"name": "ensemble_24", "kind": "ensemble", "members": 24, "steps": 10},
        # one application of the propagator in the Arnoldi stability solver
        {"name": "stability_64_fp64", "kind": "stability", "nx": 64, "ny": 65, "nz": 64, "steps": 20, "re": 2900.0},
    ]


def _steps(rng, points, most, cost):
    """Steps of a pass: up to `most`, fewer where a step costs more (cost: points times a weight)."""
    return max(3, min(most, int(LARGEST * 20 / (points * cost) * rng.uniform(0.3, 0.9))))


def _grid(rng, least, most):
    while True:
        nx, nz = rng.choice(LENGTHS), rng.choice(LENGTHS)
        ny = int(round(math.exp(rng.uniform(math.log(17), math.log(230)))))
        if least <= nx * ny * nz <= most and nx <= 8 * nz and nz <= 8 * nx:
            return nx, ny, nz


def draw(rng):
    what = rng.choice(("dns", "dns", "dns", "dns", "les", "train", "ensemble", "stability"))
    if what == "dns":
        precision = rng.choice(("mixed", "mixed", "fp64"))
        target = math.exp(rng.uniform(math.log(2e4), math.log(LARGEST / 2)))
        nx, ny, nz = _grid(rng, 0.5 * target, 1.5 * target)
        jet = rng.random() < 0.25
        return _dns(nx, ny, nz, precision, _steps(rng, nx * ny * nz, 40, 1.6 if precision == "mixed" else 4.0),
                    re=round(rng.uniform(2000.0, 6000.0), 1), dt=rng.choice((0.002, 0.0025, 0.004)),
                    ampl=rng.choice((1e-3, 1e-2)), adaptive=rng.random() < 0.3, jet=jet,
                    feedback=jet and rng.random() < 0.5)
    if what == "les":
        nx, nz = rng.choice((32, 48, 64, 96, 128)), rng.choice((32, 48, 64, 96, 128))
        ny, model = rng.randrange(25, 90), rng.choice((1, 2))
        return {"kind": "les", "nx": nx, "ny": ny, "nz": nz, "model": model, "re": round(rng.uniform(3000.0, 11000.0), 1),
                "steps": _steps(rng, nx * ny * nz, 30, 3.0 if model == 2 else 2.0)}
    if what == "train":
        return {"kind": "train", "batch": int(round(math.exp(rng.uniform(math.log(512), math.log(131072))))),
                "samples": rng.randrange(200000, 2000000), "batches": rng.randrange(1, 25)}
    if what == "ensemble":
        return {"kind": "ensemble", "members": rng.randrange(4, 31), "steps": rng.randrange(4, 13)}
    nx, nz = rng.choice((16, 24, 32, 48, 64)), rng.choice((16, 24, 32, 48, 64))
    return {"kind": "stability", "nx": nx, "ny": rng.randrange(17, 98), "nz": nz, "steps": rng.randrange(10, 31),
            "re": round(rng.uniform(2000.0, 6000.0), 1)}


# ------------------------------------------------------------ their inputs
def _field(nx, ny, nz, ampl, seed, dev):
    """data1 as (3, ny+1, nx/2+1, nz) complex128: the laminar profile and a
    discretely divergence-free disturbance that falls off as k^-2, smooth in
    y and zero on the walls."""
    g = _operators(nx, ny, nz)
    nxh, rng = nx // 2 + 1, np.random.default_rng(seed)
    c = rng.standard_normal((2, 3, nxh, nz)) + 1j * rng.standard_normal((2, 3, nxh, nz))
    c[..., nx // 2, :] = 0
    c[..., nz // 2] = 0
    c[..., 0, nz // 2 + 1:] = np.conj(c[..., 0, 1:nz // 2][..., ::-1])     # a real field
    kx, kz = g["kx"][:, None], g["kz"][None, :]
    k2 = kx * kx + kz * kz
    k2[0, 0] = 1.0
    c *= ampl * np.minimum(1.0, 1.0 / k2)
    c[..., 0, 0] = 0
    t = {n: torch.as_tensor(v, device=dev) for n, v in (("c", c), ("kx", kx), ("kz", kz), ("k2", k2))}
    y, yh, dh = (torch.as_tensor(g[n], device=dev) for n in ("y", "yh", "dh"))
    d1 = torch.zeros((3, ny + 1, nxh, nz), dtype=torch.complex128, device=dev)
    poly = torch.stack([torch.ones_like(y), y, y * y - 0.3]) * (1 - y * y) ** 2
    d1[1, :ny] = torch.einsum("mj,mab->jab", poly.to(torch.complex128), t["c"][0])
    poly = torch.stack([torch.ones_like(yh), yh, yh * yh - 0.3]) * (1 - yh * yh)
    eta = torch.einsum("mj,mab->jab", poly.to(torch.complex128), t["c"][1])[1:ny]
    dv = dh[1:ny, None, None] * (d1[1, 1:ny] - d1[1, :ny - 1])
    d1[0, 1:ny] = 1j * (-t["kz"] * eta + t["kx"] * dv) / t["k2"]
    d1[2, 1:ny] = 1j * (t["kx"] * eta + t["kz"] * dv) / t["k2"]
    d1[0, :, 0, 0] = 1 - yh * yh
    return d1


class _Run:
    """A context with the seeded field as its state, and the host arrays that take the state back."""

    def __init__(self, c, seed, dt=None, jet=None):
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        self.mixed = c.get("precision", "mixed") == "mixed"
        self.steps = c["steps"]
        grid = cf.Grid(nx, ny, nz, lx=LX, lz=LZ, stretch=STRETCH)
        self.flow = cf.ChannelFlow(grid, re=c["re"], dt=dt or c["dt"], fix_mass=1,
                                   cfl_max=0.5 if c.get("adaptive") else 0.95, dt_flag=1 if c.get("adaptive") else 0,
                                   ctrlu=0.5 if c.get("feedback") else 0.0,
                                   precision=cf.MIXED if self.mixed else cf.FP64)
        n = (ny + 1) * (nx // 2 + 1) * nz
        self.host = torch.zeros(4 * n, dtype=torch.complex128)
        if torch.cuda.is_available():
            self.host = self.host.pin_memory()
        self.d1, self.d4 = self.host[:3 * n], self.host[3 * n:]
        self.out = torch.zeros(4 * n, dtype=torch.complex64) if self.mixed else self.host
        self.d1.view(3, ny + 1, nx // 2 + 1, nz).copy_(_field(nx, ny, nz, c.get("ampl", 1e-2), seed, _device()))
        f = self.flow
        self._check(f.L.cfg_upload_state(f.h, self.d1.data_ptr(), None, self.d4.data_ptr()))
        f.remove_initial_divergence()
        f.compute_initial_pressure(0)
        if jet:
            f.set_jet(jet)

    def _check(self, r):
        if r != 0:
            raise RuntimeError("the framework returned %d" % r)

    def download(self):
        f = self.flow
        self._check(f.L.cfg_download_state(f.h, self.d1.data_ptr(), None, self.d4.data_ptr()))
        if self.mixed:
            torch.view_as_real(self.out).copy_(torch.view_as_real(self.host))
        return self.out


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _jet():
    j = cf.CfgJet()
    j.mode = 2
    j.xjet[0], j.zjet[0] = 0.3 * LX, 0.5 * LZ
    j.jetmag[0] = 0.1
    j.width, j.freq, j.frac_xbuff, j.seed = 0.2, 0.5, 0.2, 2
    return j


NET_SHAPES = ((64, 10), (64,), (64, 64), (64,), (64, 64), (64,), (6, 64), (6,))


def _network(seed):
    """Parameters of the closure network, He-normal, and the normalisation of
    its inputs and outputs: stresses around a realizable isotropic state, so
    that points pass the checks and points fall back, as with a fitted one."""
    rng = np.random.default_rng(seed + 77)
    p = [rng.standard_normal(s) * math.sqrt(2.0 / s[1]) if len(s) == 2 else 0.05 * rng.standard_normal(s)
         for s in NET_SHAPES]
    p = np.concatenate([a.ravel() for a in p]).astype(np.float32)
    return p, {"in_shift": [0.0] * 9 + [0.5], "in_scale": [0.5, 3.0, 0.5, 0.5, 0.5, 0.5, 0.5, 1.0, 0.5, 0.3],
               "out_shift": [1e-3, 1e-3, 1e-3, 0.0, 0.0, 0.0], "out_scale": [2e-4] * 6}


def _training(c, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((c["samples"], 10), dtype=np.float32)
    w = rng.standard_normal((10, 6), dtype=np.float32) * 0.3
    t = np.tanh(x @ w) + 0.1 * rng.standard_normal((c["samples"], 6), dtype=np.float32)
    idx = rng.integers(0, c["samples"], (c["batches"], c["batch"]), dtype=np.int32)
    return x, t.astype(np.float32), idx


def _member(c, m):
    """Member m of an ensemble: its grid, Reynolds number and jet."""
    nx, ny, nz = ENS_GRIDS[m % 3]
    return {"nx": nx, "ny": ny, "nz": nz, "steps": c["steps"], "re": 2000.0 + 37.0 * m % 1000.0, "dt": 0.0025,
            "jet": m % 2 == 1}


def _propagated(c, seed):
    rng = np.random.default_rng(seed)
    return np.asfortranarray(rng.standard_normal((c["nx"], c["nz"], c["ny"] + 1, 3)))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dns":
        return _Run(case, seed, jet=_jet() if case["jet"] else None), kind
    if kind == "les":
        r = _Run(dict(case, precision="mixed"), seed, dt=0.002)
        if case["model"] == 2:
            p, norm = _network(seed)
            r.flow.set_les(2, mlp=cf.Mlp(params=p), **norm)
        else:
            r.flow.set_les(1)
        return r, kind
    if kind == "train":
        dev = _device()
        x, t, idx = _training(case, seed)
        return {"net": cf.Mlp(params=_network(seed)[0]), "x": torch.as_tensor(x, device=dev),
                "t": torch.as_tensor(t, device=dev), "idx": torch.as_tensor(idx, device=dev)}, kind
    if kind == "ensemble":
        runs = []
        for m in range(case["members"]):
            c = _member(case, m)
            runs.append(_Run(c, seed + 1000 + m, jet=_jet() if c["jet"] else None))
        return {"runs": runs, "ens": cf.Ensemble([r.flow for r in runs], autotune=False), "steps": case["steps"]}, kind
    grid = cf.Grid(case["nx"], case["ny"], case["nz"], lx=LX, lz=LZ, stretch=STRETCH)
    flow = cf.ChannelFlow(grid, re=case["re"], dt=0.01, fix_mass=1, precision=cf.FP64)
    base = np.zeros((case["ny"] + 1, 3), order="F")
    base[:, 0] = 1 - grid.yh ** 2
    flow.set_baseflow(base)
    return {"flow": flow, "v": _propagated(case, seed), "steps": case["steps"]}, kind


def run(state):
    s, kind = state
    if kind in ("dns", "les"):
        s.flow.timestep(s.steps)
        return s.download()
    if kind == "train":
        net, idx = s["net"], s["idx"]
        x, t, n = s["x"].data_ptr(), s["t"].data_ptr(), idx.shape[0]
        for k in range(n):
            net.accumulate_grad(x, t, idx[k].data_ptr(), idx.shape[1])
        grads, loss = net.grads()       # as a program logs its loss
        net.adam_step(1e-3)
        return {"gradient": grads, "loss": np.array([loss], np.float32), "params": net.get_params()}
    if kind == "ensemble":
        s["ens"].timestep(s["steps"])
        s["ens"].synchronize()
        return [r.download() for r in s["runs"]]
    return s["flow"].arnoldi_matvec(s["v"], s["steps"])


# ------------------------------------------------------------ what it takes
def _step_work(nx, ny, nz, real):
    """Bytes and operations of one time step: in each of three substeps the
    transforms read the velocity and write the nonlinear term, and the solves
    read that, the accumulator and the pressure and write velocity,
    accumulator and pressure."""
    nxh, n1, nx2, nz2 = nx // 2 + 1, ny + 1, 3 * nx // 2, 3 * nz // 2
    nf = nxh * nz * n1
    fft = n1 * ((3 + 6) * nxh * 5.0 * nz2 * math.log2(nz2) + (3 + 8) * nz2 * 2.5 * nx2 * math.log2(nx2))
    return 3 * 20.0 * nf * 2 * real, 3 * (fft + n1 * nz2 * nx2 * 60.0 + nf * 300.0)


def work(case):
    kind = case["kind"]
    if kind == "train":
        b, s = case["batch"], case["batches"]
        net = 10 * 64 + 2 * 64 * 64 + 6 * 64
        return {"bytes": s * (b * (16 * 4.0 + 4.0) + 7 * 4.0 * net), "flops": s * 6.0 * b * net}
    if kind == "ensemble":
        parts = [work(dict(_member(case, m), kind="dns")) for m in range(case["members"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nx, ny, nz, n = case["nx"], case["ny"], case["nz"], case["steps"]
    fp64 = kind == "stability" or case.get("precision") == "fp64"
    b, f = _step_work(nx, ny, nz, 8 if fp64 else 4)
    back = 16.0 * (nx * nz * (ny + 1) * 3 if kind == "stability" else (nx // 2 + 1) * nz * (ny + 1) * 4)
    pts = 2.25 * nx * nz * (ny - 1)
    if kind == "les":
        f += 3 * pts * (100.0 + (2.0 * 9216 if case["model"] == 2 else 0.0))
    return {"bytes": n * b + back, "flops": n * f}


# ------------------------------------------------------- the same, in 64 bits
RKA = (0.0, -17.0 / 60.0, -5.0 / 12.0)
RKB = (8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0)
RKC = (29.0 / 96.0, -3.0 / 40.0, 1.0 / 6.0)
RKD = (37.0 / 160.0, 5.0 / 24.0, 1.0 / 6.0)
RKA, RKB, RKC, RKD = ([float(np.float32(v)) for v in t] for t in (RKA, RKB, RKC, RKD))


def _operators(nx, ny, nz):
    """The staggered grid of the channel and its difference operators (numpy)."""
    xi = 2.0 * np.arange(ny) / (ny - 1) - 1.0
    y = np.tanh(STRETCH * xi) / np.tanh(STRETCH)
    yh = np.concatenate([y[:1], 0.5 * (y[:-1] + y[1:]), y[-1:]])
    hh = np.concatenate([[y[1] - y[0]], y[1:] - y[:-1], [y[-1] - y[-2]]])
    hn = yh[1:] - yh[:-1]
    dh, dn = 1 / hh, 1 / hn
    a, b, c, d = hn[0], hn[1], hn[ny - 2], hn[ny - 1]
    dm = np.array([[-dn[0] * (2 * a + b) / (a + b), dn[0] * dn[1] * (a + b), -dn[1] * a / (a + b)],
                   [dn[ny - 2] * d / (c + d), -dn[ny - 1] * dn[ny - 2] * (d + c), dn[ny - 1] * (2 * d + c) / (d + c)]])
    d2n, d2h = np.zeros((ny, 3)), np.zeros((ny + 1, 3))
    i = np.arange(1, ny - 1)
    d2n[i] = np.stack([dn[i] * dh[i], -dn[i] * dh[i] - dn[i] * dh[i + 1], dn[i] * dh[i + 1]], 1)
    d2h[i] = np.stack([dh[i] * dn[i - 1], -dh[i] * dn[i - 1] - dh[i] * dn[i], dh[i] * dn[i]], 1)
    d2h[1] = -dh[1] * dm[0, 0], -dh[1] * dn[1] - dh[1] * dm[0, 1], dh[1] * dn[1] - dh[1] * dm[0, 2]
    e = ny - 1
    d2h[e] = dh[e] * dn[e - 1] + dh[e] * dm[1, 0], -dh[e] * dn[e - 1] + dh[e] * dm[1, 1], dh[e] * dm[1, 2]
    d2h[0], d2n[0], d2n[ny - 1], d2h[ny] = d2h[1], d2n[1], d2n[ny - 2], d2h[ny - 1]
    dyh = hh.copy()
    dyh[0] = dyh[ny] = 0
    dy = np.concatenate([[0.5 * hh[1]], 0.5 * (hh[1:ny - 1] + hh[2:ny]), [0.5 * hh[ny - 1]], [0.0]])
    kz = np.fft.fftfreq(nz, 1.0 / nz) * (2 * math.pi / LZ)
    kz[nz // 2] = abs(kz[nz // 2])
    return {"y": y, "yh": yh, "hn": hn, "dh": dh, "dn": dn, "dm": dm, "d2h": d2h, "d2n": d2n, "dyh": dyh, "dy": dy,
            "iu1": 0.5 * hh[:ny] / hn, "iu2": 0.5 * hh[1:] / hn, "kx": np.arange(nx // 2 + 1) * (2 * math.pi / LX),
            "kz": kz}


class _Exact:
    """The time step in 64 bits.  Fields are (plane, kx, kz) and (plane, z, x)."""

    def __init__(self, nx, ny, nz, re, dt, cfl_max=0.95, adaptive=False, ctrlu=0.0, jet=False, base=None):
        self.nx, self.ny, self.nz, self.re, self.dt = nx, ny, nz, re, dt
        self.nxh, self.nx2, self.nz2 = nx // 2 + 1, 3 * nx // 2, 3 * nz // 2
        self.cfl_max, self.adaptive, self.ctrlu, self.jet, self.les = cfl_max, adaptive, ctrlu, jet, None
        self.dev = _device()
        self.h = _operators(nx, ny, nz)
        self.g = {k: torch.as_tensor(v, device=self.dev) for k, v in self.h.items()}
        self.ikx = (1j * self.g["kx"]).view(-1, 1)
        self.ikz = (1j * self.g["kz"]).view(1, -1)
        self.k2 = (self.g["kx"].view(-1, 1) ** 2 + self.g["kz"].view(1, -1) ** 2)
        self.base = None if base is None else torch.as_tensor(base, device=self.dev)
        self.t, self.p_grad = 0.0, -2.0 / re
        self.dum = np.zeros(ny)
        z = lambda *s: torch.zeros(s, dtype=torch.complex128, device=self.dev)  # noqa: E731
        self.bot, self.top = z(3, self.nxh, nz), z(3, self.nxh, nz)
        self.cru, self.p = z(3, ny + 1, self.nxh, nz), z(ny + 1, self.nxh, nz)
        self.v = None

    # transforms of planes, 3/2 dealiased (Nyquist modes split, then folded)
    def c2r(self, c):
        nz, nz2, h = self.nz, self.nz2, self.nz // 2
        q = torch.zeros(c.shape[:-1] + (nz2,), dtype=c.dtype, device=c.device)
        q[..., :h] = c[..., :h]
        q[..., nz2 - h + 1:] = c[..., h + 1:]
        q[..., h] = 0.5 * c[..., h]
        q[..., nz2 - h] = 0.5 * c[..., h].conj()
        q[..., -1, :] *= 0.5
        q = torch.fft.ifft(q, dim=-1, norm="forward").transpose(-1, -2).contiguous()
        q[..., 0].imag.zero_()
        return torch.fft.irfft(q, n=self.nx2, dim=-1, norm="forward")

    def _fold(self, f):
        nz, h = self.nz, self.nz // 2
        o = torch.zeros(f.shape[:-1] + (nz,), dtype=f.dtype, device=f.device)
        o[..., :h] = f[..., :h]
        o[..., h] = f[..., h] + f[..., self.nz2 - h].conj()
        o[..., h + 1:] = f[..., self.nz2 - h + 1:]
        o = o / (self.nx2 * self.nz2)
        o[..., -1, :] *= 2
        return o

    def _rows(self, f):
        return torch.fft.rfft(f, dim=-1)[..., :self.nxh].transpose(-1, -2)

    def r2c(self, f):
        return self._fold(torch.fft.fft(self._rows(f), dim=-1))

    def div(self, fx, fy, fz):
        a = torch.fft.fft(self._rows(fy) + self.ikx * self._rows(fx), dim=-1)
        return self._fold(a) + self.ikz * self.r2c(fz)

    def stresses(self, U, V, W, k):
        """Subgrid stresses (11, 22, 33, 12, 13, 23) at the interior yh planes k0 = k (0-based array)."""
        g, hx, hz = self.g, LX / self.nx2, LZ / self.nz2
        ddx = lambda f: (torch.roll(f, -1, -1) - torch.roll(f, 1, -1)) / (2 * hx)  # noqa: E731
        ddz = lambda f: (torch.roll(f, -1, -2) - torch.roll(f, 1, -2)) / (2 * hz)  # noqa: E731
        col = lambda v: v.view(-1, 1, 1)  # noqa: E731
        idy = col(1 / (g["yh"][k + 1] - g["yh"][k - 1]))
        vc = 0.5 * (V[k - 1] + V[k])
        G = [[ddx(U[k]), (U[k + 1] - U[k - 1]) * idy, ddz(U[k])],
             [ddx(vc), (V[k] - V[k - 1]) * col(g["dh"][k]), ddz(vc)],
             [ddx(W[k]), (W[k + 1] - W[k - 1]) * idy, ddz(W[k])]]
        tr = (G[0][0] + G[1][1] + G[2][2]) / 3
        S = [G[0][0] - tr, G[1][1] - tr, G[2][2] - tr, 0.5 * (G[0][1] + G[1][0]), 0.5 * (G[0][2] + G[2][0]),
             0.5 * (G[1][2] + G[2][1])]
        dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + 2 * (a[3] * b[3] + a[4] * b[4] + a[5] * b[5])  # noqa: E731
        utau = math.sqrt(0.5 * (abs(self.dum[0]) + abs(self.dum[-1])) / self.re)
        yp = (1 - g["yh"][k].abs()) * utau * self.re
        delta = (LX / self.nx * LZ / self.nz * (g["y"][k] - g["y"][k - 1])) ** (1.0 / 3.0)
        nut = col(0.1 * delta * (1 - torch.exp(-yp / 25.0))) ** 2 * torch.sqrt(2 * dot(S, S))
        ev = [-2 * nut * s for s in S]
        if self.les[0] == 1:
            return ev
        _, params, norm = self.les
        sgn = col(torch.where(g["yh"][k] > 0, -1.0, 1.0).to(torch.float64))
        wall = col(1 - g["yh"][k].abs()).expand_as(tr)
        f = [G[0][0], sgn * G[0][1], G[0][2], sgn * G[1][0], G[1][1], sgn * G[1][2], G[2][0], sgn * G[2][1], G[2][2], wall]
        f = torch.stack([(a - s) / c for a, s, c in zip(f, norm["in_shift"], norm["in_scale"])], -1)
        o = _mlp([a.to(self.dev) for a in params], f)
        t = [s + c * o[..., i] for i, (s, c) in enumerate(zip(norm["out_shift"], norm["out_scale"]))]
        t[3], t[5] = sgn * t[3], sgn * t[5]
        det = (t[0] * (t[1] * t[2] - t[5] * t[5]) - t[3] * (t[3] * t[2] - t[5] * t[4])
               + t[4] * (t[3] * t[5] - t[1] * t[4]))
        ok = ((t[0] >= 0) & (t[1] >= 0) & (t[2] >= 0) & (t[3] ** 2 <= t[0] * t[1]) & (t[4] ** 2 <= t[0] * t[2])
              & (t[5] ** 2 <= t[1] * t[2]) & (det >= 0) & (-dot(t, S) >= 0))
        return [torch.where(ok, a, b) for a, b in zip(t, ev)]

    def nonlinear(self, rk, step=1):
        """The divergence of the momentum fluxes of self.v, and the CFL rule."""
        ny, g, half = self.ny, self.g, 0.5
        out = torch.zeros_like(self.v)
        U, V, W = (torch.empty((ny + 1, self.nz2, self.nx2), dtype=torch.float64, device=self.dev) for _ in range(3))
        for q, f in enumerate((U, V, W)):
            for j in range(0, ny + 1, 16):
                f[j:j + 16] = self.c2r(self.v[q, j:j + 16])
        S = None
        if self.les:
            S = torch.zeros((6, ny + 1, self.nz2, self.nx2), dtype=torch.float64, device=self.dev)
            for j in range(1, ny, 16):
                k = torch.arange(j, min(j + 16, ny), device=self.dev)
                for c, s in enumerate(self.stresses(U, V, W, k)):
                    S[c, k] = s
        B = self.base
        cfl = 0.0
        for j in range(1, ny, 16):        # planes k = 2..ny of the reference are 1..ny-1 here
            k = torch.arange(j, min(j + 16, ny), device=self.dev)
            col = lambda v: v.view(-1, 1, 1)  # noqa: E731
            first, last = col(k == 1), col(k == ny - 1)
            u, v, w = U[k], V[k], W[k]
            um, vm, wm, up, wp = U[k - 1], V[k - 1], W[k - 1], U[k + 1], W[k + 1]
            vp = torch.where(last, v, V[torch.clamp(k + 1, max=ny - 1)])
            dh, dn = col(g["dh"][k]), col(g["dn"][k])
            i1, i2 = col(g["iu1"][k]), col(g["iu2"][k])
            lo = lambda a, b: torch.where(first, a, half * (a + b))  # noqa: E731  onto plane k-1
            hi = lambda a, b: torch.where(last, b, half * (a + b))  # noqa: E731  onto plane k
            v0, v1 = half * (vm + v), half * (v + vp)
            if B is None:
                fu = dh * (v * hi(u, up) - vm * lo(um, u))
                fw = dh * (v * hi(w, wp) - vm * lo(wm, w))
                uu, uw, ww = u * u, u * w, w * w
                vu, vw = v * (i1 * u + i2 * up), v * (i1 * w + i2 * wp)
                vv = dn * (v1 * v1 - v0 * v0)
            else:
                b0, bm, bp = ([col(B[n, c]) for c in range(3)] for n in (k, k - 1, k + 1))
                flux = lambda f, fm, fp, c: dh * (  # noqa: E731
                    b0[1] * hi(f, fp) + v * hi(b0[c], bp[c]) - bm[1] * lo(fm, f) - vm * lo(bm[c], b0[c]))
                fu, fw = flux(u, um, up, 0), flux(w, wm, wp, 2)
                uu, uw, ww = 2 * b0[0] * u, b0[2] * u + w * b0[0], 2 * b0[2] * w
                vu = b0[1] * (i1 * u + i2 * up) + v * (i1 * b0[0] + i2 * bp[0])
                vw = b0[1] * (i1 * w + i2 * wp) + v * (i1 * b0[2] + i2 * bp[2])
                vv = dn * (v1 * (b0[1] + bp[1]) - v0 * (bm[1] + b0[1]))
            if S is not None:
                s, sm, sp = S[:, k], S[:, k - 1], S[:, k + 1]
                zero = torch.zeros_like(u)
                y1 = lambda c: torch.where(last, zero, half * (s[c] + sp[c]))  # noqa: E731
                y0 = lambda c: torch.where(first, zero, half * (sm[c] + s[c]))  # noqa: E731
                uu, uw, ww = uu + s[0], uw + s[4], ww + s[2]
                fu, fw = fu + dh * (y1(3) - y0(3)), fw + dh * (y1(5) - y0(5))
                vu, vw = vu + i1 * s[3] + i2 * sp[3], vw + i1 * s[5] + i2 * sp[5]
                vv = vv + dn * (sp[1] - s[1])
            out[0, k] = self.div(uu, fu, uw)
            out[2, k] = self.div(uw, fw, ww)
            o = self.div(vu, vv, vw)
            o[k == ny - 1] = 0
            out[1, k] = o
            if rk == 0:
                m = lambda f: f.abs().amax((1, 2))  # noqa: E731
                a, b, c = m(u + up), m(v), m(w + wp)
                if B is not None:
                    a, b, c = (torch.maximum(x, z.abs().view(-1)) for x, z in
                               ((a, b0[0] + bp[0]), (b, b0[1]), (c, b0[2] + bp[2])))
                hmin = torch.minimum(g["hn"][k], g["hn"][k - 1])
                cfl = max(cfl, float((half * a * self.nx / (0.55 * LX) + b / (1.73 * hmin)
                                      + half * c * self.nz / (0.55 * LZ)).max()) * self.dt)
        if rk == 0 and step >= 0 and self.adaptive:
            d = self.dt * self.cfl_max / cfl
            self.dt = min(d, self.dt + (d - self.dt) * self.dt / (1 + self.dt))
        return out

    # columns: (plane, kx, kz)
    def d2(self, f, n, name):
        d, o = self.g[name].view(-1, 3, 1, 1), torch.zeros_like(f)
        o[1:n - 1] = d[1:n - 1, 0] * f[:n - 2] + d[1:n - 1, 1] * f[1:n - 1] + d[1:n - 1, 2] * f[2:n]
        o[0] = d[0, 0] * f[0] + d[0, 1] * f[1] + d[0, 2] * f[2]
        o[n - 1] = d[n - 1, 0] * f[n - 3] + d[n - 1, 1] * f[n - 2] + d[n - 1, 2] * f[n - 1]
        return o

    @staticmethod
    def tri(a, b, c, f):
        """Thomas sweeps: a, b, c lists of rows, f (rows, [rhs,] kx, kz) in place."""
        n, cc = len(b), [None] * len(b)
        r = 1 / b[0]
        cc[0] = c[0] * r
        f[0] = f[0] * r
        for i in range(1, n):
            r = 1 / (b[i] - a[i] * cc[i - 1])
            cc[i] = c[i] * r
            f[i] = (f[i] - a[i] * f[i - 1]) * r
        for i in range(n - 2, -1, -1):
            f[i] -= cc[i] * f[i + 1]
        return f

    def helmholtz(self, f, n, name, alpha, vis, bot, top):
        d, one = self.h[name], torch.ones_like(alpha)
        f[0], f[n - 1] = bot, top
        a = [0.0] + [-vis * float(d[i, 0]) for i in range(1, n - 1)] + [0.0]
        b = [one] + [alpha - vis * float(d[i, 1]) for i in range(1, n - 1)] + [one]
        c = [0.0] + [-vis * float(d[i, 2]) for i in range(1, n - 1)] + [0.0]
        return self.tri(a, b, c, f[:n])

    def strip(self, cv, coef):
        """Removes the divergence of cv; returns the correction potential."""
        ny, h, k2 = self.ny, self.h, self.k2.clone()
        k2[0, 0] = 1.0
        dh, dn, dm = self.g["dh"].view(-1, 1, 1), self.g["dn"].view(-1, 1, 1), h["dm"]
        p = torch.zeros_like(cv[0])
        p[1:ny] = (self.ikx * cv[0, 1:ny] + dh[1:ny] * (cv[1, 1:ny] - cv[1, :ny - 1]) + self.ikz * cv[2, 1:ny]) / coef
        one = torch.ones_like(k2)
        lo, up = h["dh"][1:ny] * h["dn"][:ny - 1], h["dh"][1:ny] * h["dn"][1:ny]
        a = [0.0] + [float(v) for v in lo] + [-float(h["dn"][ny - 1])]
        b = [-float(h["dn"][0]) * one] + [-float(x) - float(z) - k2 for x, z in zip(lo, up)] + [float(h["dn"][ny - 1]) * one]
        c = [float(h["dn"][0])] + [float(v) for v in up] + [0.0]
        self.tri(a, b, c, p)
        p[0] = (-dm[0, 1] * p[1] - dm[0, 2] * p[2]) / dm[0, 0]
        p[ny] = (-dm[1, 0] * p[ny - 2] - dm[1, 1] * p[ny - 1]) / dm[1, 2]
        p[:, 0, 0] = 0
        self.subtract(cv, p, coef)
        return p

    def subtract(self, cv, p, coef):
        ny, dn = self.ny, self.g["dn"].view(-1, 1, 1)
        cv[0, 1:ny] -= coef * self.ikx * p[1:ny]
        cv[2, 1:ny] -= coef * self.ikz * p[1:ny]
        cv[1, 1:ny - 1] -= coef * dn[1:ny - 1] * (p[2:ny] - p[1:ny - 1])

    def viscous(self, cv, f, vis):
        for q, (n, name) in enumerate(((self.ny + 1, "d2h"), (self.ny, "d2n"), (self.ny + 1, "d2h"))):
            cv[q, :n] += vis * (self.d2(f[q], n, name)[:n] - self.k2 * f[q, :n])

    def set_jet(self, rk):
        nx = self.nx
        x = np.arange(nx) * LX / nx
        a, end, edge = 0.8 * LX, 0.9 * LX, 0.025 * LX       # suction that balances the jet
        ramp = lambda s: 1 / (1 + np.exp(1 / s + 1 / (s - 1)))  # noqa: E731
        f = np.zeros(nx)
        for i, xc in enumerate(x):
            if a < xc < end:
                f[i] = ramp((xc - a) / edge) if xc < a + edge else ramp((end - xc) / edge) if xc > end - edge else 1.0
        time = self.t + self.dt * sum(RKC[r] + RKD[r] for r in range(rk + 1))
        d = np.abs(x - 0.3 * LX)
        d = np.minimum(d, LX - d)
        v = 0.1 * 0.5 * (1 + math.sin(2 * math.pi * 0.5 * time)) * np.exp(-(d / 0.2) ** 2)
        cs, cj = np.fft.rfft(f) / nx, np.fft.rfft(v) / nx
        self.bot[1], self.top[1] = 0, 0
        self.bot[1, :, 0] = torch.as_tensor(cj - cj[0].real / cs[0].real * cs, device=self.dev)

    def solve(self, nl, rk):
        ny, dt, cru = self.ny, self.dt, self.cru
        vis, press, coef = RKD[rk] * (dt / self.re), (RKC[rk] + RKD[rk]) * dt, RKB[rk] * dt
        if self.jet:
            self.set_jet(rk)
        cv = cru - coef * nl
        if rk == 0:
            self.viscous(cv, cru, RKC[0] * (dt / self.re))
            self.subtract(cv, self.p, press)        # the mean mode's pressure is zero
        flux = float((self.g["dyh"][1:ny] * -nl[0, 1:ny, 0, 0].real).sum())
        self.p_grad = -flux + 0.5 * (self.dum[ny - 1] - self.dum[0]) / self.re
        cv[0, :, 0, 0] -= press * self.p_grad
        alpha = 1 + vis * self.k2
        uw = torch.stack([cv[0], cv[2]], 1)
        uw = self.helmholtz(uw, ny + 1, "d2h", alpha, vis, self.bot[::2], self.top[::2])
        cv[0], cv[2] = uw[:, 0], uw[:, 1]
        cv[1, :ny] = self.helmholtz(cv[1].clone(), ny, "d2n", alpha, vis, self.bot[1], self.top[1])
        cv[1, ny] = 0
        cv[1, :ny, 0, 0] = self.bot[1, 0, 0]
        ch = self.strip(cv, press)
        self.p = self.p + alpha * ch - vis * self.d2(ch, ny + 1, "d2h")
        self.p[:, 0, 0] = 0
        self.v = cv
        if rk < 2:
            self.cru = cv - dt * RKA[rk + 1] * nl
            self.viscous(self.cru, cv, (dt / self.re) * RKC[rk + 1])
            self.subtract(self.cru, self.p, (RKC[rk + 1] + RKD[rk + 1]) * dt)
        else:
            self.cru = cv.clone()
        self.shear()

    def shear(self):
        u, dm, ny = self.v[0, :, 0, 0].real.cpu().numpy(), self.h["dm"], self.ny
        self.dum = np.zeros(ny)
        self.dum[0], self.dum[-1] = dm[0] @ u[:3], dm[1] @ u[ny - 2:]

    def start(self, v, keep_mean=True):
        """define_initial_field for a given velocity: its divergence removed, its pressure."""
        self.v = v
        if keep_mean:
            v0 = self.v[1, :, 0, 0].clone()
            self.strip(self.v, 1.0)
            self.v[1, :, 0, 0] = v0
            self.v[1, 1:self.ny, 0, 0] = v0[0]
            self.shear()
        self.cru = self.v.clone()
        r = -self.nonlinear(2, -1)
        self.viscous(r, self.v, 1.0 / self.re)
        self.p = self.strip(r, 1.0)

    def walls(self):
        self.bot.zero_()
        self.top.zero_()
        if self.ctrlu:
            ny, dm = self.ny, self.h["dm"]
            u = self.c2r(self.v[0][[1, 2, ny - 1, ny - 2]])
            lo = (dm[0, 1] * u[0] + dm[0, 2] * u[1] - 2.0) / (self.ctrlu - dm[0, 0])
            hi = -(dm[1, 1] * u[2] + dm[1, 0] * u[3] + 2.0) / (self.ctrlu + dm[1, 2])
            self.bot[0], self.top[0] = self.r2c(lo), self.r2c(hi)

    def steps(self, n):
        for _ in range(n):
            if self.base is None:
                self.walls()
            for rk in range(3):
                self.solve(self.nonlinear(rk), rk)
            self.t += self.dt

    def outputs(self):
        return torch.cat([self.v.reshape(-1), self.p.permute(1, 2, 0).reshape(-1)])


def _mlp(params, x):
    for layer in range(4):
        x = x @ params[2 * layer].T + params[2 * layer + 1]
        if layer < 3:
            x = torch.nn.functional.gelu(x, approximate="tanh")
    return x


def _params64(flat):
    out, at = [], 0
    for s in NET_SHAPES:
        n = int(np.prod(s))
        out.append(torch.as_tensor(flat[at:at + n].astype(np.float64).reshape(s)))
        at += n
    return out


def _exact_steps(c, seed, mixed, dt, les=None, **kw):
    e = _Exact(c["nx"], c["ny"], c["nz"], c["re"], dt, **kw)
    v = _field(c["nx"], c["ny"], c["nz"], c.get("ampl", 1e-2), seed, e.dev)
    if mixed:       # what an FP32 state holds of it
        mean = v[:, :, 0, 0].clone()
        v = v.to(torch.complex64).to(torch.complex128)
        v[:, :, 0, 0] = mean
    e.start(v)
    e.les = les
    e.steps(c["steps"])
    return e.outputs()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dns", "les"):
        cost = case["steps"] * case["nx"] * case["nz"] * case["ny"]
        if cost > 6e8:       # over about 20 seconds
            return None
        if kind == "dns":
            return _exact_steps(case, seed, case["precision"] == "mixed", case["dt"],
                                cfl_max=0.5 if case["adaptive"] else 0.95, adaptive=case["adaptive"],
                                ctrlu=0.5 if case["feedback"] else 0.0, jet=case["jet"])
        les = (1,)
        if case["model"] == 2:
            p, norm = _network(seed)
            les = (2, _params64(p), {k: [float(np.float32(a)) for a in v] for k, v in norm.items()})
        return _exact_steps(case, seed, True, 0.002, les=les)
    if kind == "train":
        dev = _device()
        x, t, idx = (torch.as_tensor(a, device=dev) for a in _training(case, seed))
        p = [a.to(dev).requires_grad_() for a in _params64(_network(seed)[0])]
        g, total = [torch.zeros_like(a) for a in p], 0.0
        for at in idx.long():
            loss = ((_mlp(p, x[at].double()) - t[at].double()) ** 2).mean()
            for a, d in zip(g, torch.autograd.grad(loss, p)):
                a += d
            total += float(loss)
        with torch.no_grad():       # the first Adam update: its moments are the gradient and its square
            p = [a - 1e-3 * d / (d.abs() + 1e-8) for a, d in zip(p, g)]
        flat = lambda ts: torch.cat([a.detach().reshape(-1) for a in ts]).cpu().numpy()  # noqa: E731
        return {"gradient": flat(g), "loss": np.array([total]), "params": flat(p)}
    if kind == "ensemble":
        out = []
        for m in range(case["members"]):
            c = _member(case, m)
            # every grid with and without the jet; all members would take too long
            out.append(None if m >= 6 else _exact_steps(c, seed + 1000 + m, True, c["dt"], jet=c["jet"]))
        return out
    e = _Exact(case["nx"], case["ny"], case["nz"], case["re"], 0.01, base=_baseflow(case))
    v = torch.as_tensor(np.ascontiguousarray(_propagated(case, seed).T), device=e.dev)      # (3, plane, z, x)
    scale = 1e-8 / float(v.abs().max())
    wgt = torch.stack([e.g["dyh"], e.g["dy"], e.g["dyh"]]).view(3, -1, 1, 1)
    c = torch.fft.fft(torch.fft.rfft(v, dim=-1).transpose(-1, -2), dim=-1) / (case["nx"] * case["nz"])
    c = torch.where(wgt > 0, c * (scale / torch.where(wgt > 0, wgt, torch.ones_like(wgt)).sqrt()), torch.zeros_like(c))
    e.p_grad = 0.0
    e.start(c, keep_mean=False)
    e.steps(case["steps"])
    q = torch.fft.ifft(e.v * (wgt.sqrt() / scale), dim=-1, norm="forward").transpose(-1, -2).contiguous()
    q[..., 0].imag.zero_()
    q[..., -1].imag.zero_()
    w = torch.fft.irfft(q, n=case["nx"], dim=-1, norm="forward")
    return np.ascontiguousarray(w.cpu().numpy()).T


def _baseflow(case):
    b = np.zeros((case["ny"] + 1, 3))
    b[:, 0] = 1 - _operators(case["nx"], case["ny"], case["nz"])["yh"] ** 2
    return b
