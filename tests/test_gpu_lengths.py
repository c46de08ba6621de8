"""The register-FFT transform lengths 36, 54, 108, 162, 216, 324 and 432 in x
and in z (grids with nx or nz of 24, 36, 72, 108, 144, 216 and 288): the
nonlinear term with a fringe and its CFL number, and the linearized nonlinear
term, against the shared-memory FFT path (CHANFLOW_GENERIC_FFT), which every
length takes and which the oracle tests cover, for every flux tile a context
accepts.

FP64: two orderings of the same transforms and products agree to 1e-12
(relative L2, the bar of the oracle comparisons per routine).  Mixed
precision: the rounding of the FP32 products reaches the result multiplied by
the wavenumber, up to 1e-5 of it at these lengths on either path, so the bar
is the generic path's own distance from FP64: the register path may be no
further from it than 1.5 times that (CFL number: 1e-6, the bar of the oracle
comparison).  z rows that no tile divides (54, 162
rows) and row counts of 4 modulo 8 (36, 108, 324) exercise the last block of
the x stage."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(24, 36), (36, 24), (72, 16), (16, 72), (108, 24), (24, 108), (144, 36), (36, 144), (216, 16), (16, 216),
         (288, 16), (16, 288)]
KEYS = ("CHANFLOW_GENERIC_FFT", "CHANFLOW_NO_MEAN_SPLIT")


def terms(cf, nx, nz, prec, env, tiles=None):
    saved = {k: os.environ.pop(k, None) for k in KEYS}
    os.environ.update(env)
    try:
        f = cf.ChannelFlow(cf.Grid(nx, 10, nz, stretch=1.5), re=2500.0, dt=0.004, precision=prec)
    finally:
        for k in KEYS:
            os.environ.pop(k, None)
            if saved[k] is not None:
                os.environ[k] = saved[k]
    f.init_buffer(4.0, xfringe=1, zfringe=1, frac_xbuff=0.2, buff_xrise=0.06, buff_xfall=0.03, frac_zbuff=0.15)
    f.define_initial_field(10, seed=21, ampl=5e-2)
    if tiles:
        f.set_tiles(tiles)
    f.nonlinear(1, 1)
    out = [f.download_state()[0]]
    cfl = f.scalars()["cfl_max"]
    f.define_initial_field(10, seed=22, ampl=5e-2)
    base = np.zeros((11, 3), order="F")
    base[:, 0] = 1 - f.grid.yh ** 2
    f.set_baseflow(base)
    # the linearized products have no 8-row tile: the x lengths of the other
    # paths (here 24: nx 16) refuse it, the new ones take fewer rows
    if not (tiles and tiles[1] == 8 and nx == 16):
        f.nonlinear_linearized(1, 1)
        out.append(f.download_state()[0])
    assert f.status() == 0
    f.close()
    return out, cfl


TILES = (None, (2, 2, 1, 1), (2, 4, 8, 8))


def dist(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nx,nz", SIZES)
def test_length_matches_generic_transforms(cf, nx, nz):
    ref, cfl = terms(cf, nx, nz, 0, {"CHANFLOW_GENERIC_FFT": "1"})
    for tiles in TILES:
        got, c = terms(cf, nx, nz, 0, {}, tiles)
        assert abs(c - cfl) < 1e-12 * cfl, tiles
        for a, b in zip(got, ref):
            assert dist(a, b) < 1e-12, tiles
    whole = {"CHANFLOW_NO_MEAN_SPLIT": "1"}
    bar = [1.5 * dist(a, b) for a, b in zip(terms(cf, nx, nz, 1, dict(whole, CHANFLOW_GENERIC_FFT="1"))[0], ref)]
    for env in (whole, {}):
        for tiles in TILES + ((2, 8, 3, 3),):
            got, c = terms(cf, nx, nz, 1, env, tiles)
            assert abs(c - cfl) < 1e-6 * cfl, (env, tiles)
            for a, b, t in zip(got, ref, bar):
                assert dist(a, b) < t, (env, tiles)


def test_lengths_keep_their_refusals(cf):
    """The LES mode and the batched ensemble layout stay with the lengths they list."""
    grid = cf.Grid(72, 10, 72, stretch=1.5)
    f = [cf.ChannelFlow(grid, re=2500.0, dt=0.004, precision=1) for _ in range(2)]
    with pytest.raises(cf.ChanflowError):
        f[0].set_les(1)
    ens = cf.Ensemble(f, autotune=False)
    assert not ens.batched
    with pytest.raises(cf.ChanflowError):
        cf.Ensemble(f, autotune=False, batched=True)
    ens.close()
