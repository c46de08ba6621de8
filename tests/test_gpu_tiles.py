"""Launch tiles where a context's other products lack one of them: the flux
kernel has blocks of 8 z rows (FP32) for the nonlinear products only.  A
context takes the LES mode and linearized steps whatever chose the tile --
the caller, a context's own tiles put back, the tuner or an ensemble -- and
their states are those of the 4-row tile, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def flow_of(cf, nx, ny=17, nz=32, prec=1):
    f = cf.ChannelFlow(cf.Grid(nx, ny, nz, stretch=1.5), re=3000.0, dt=0.002, precision=prec)
    f.define_initial_field(10, seed=2, ampl=5e-2)
    return f


def steps(f, what):
    if what == "les":
        f.set_les(1)
        f.timestep(3)
    else:
        base = np.zeros((f.ny + 1, 3), order="F")
        base[:, 0] = 1 - f.grid.yh ** 2
        f.set_baseflow(base)
        f.timestep_linearized(3)
    assert f.status() == 0
    return f.download_state()


@pytest.mark.parametrize("what", ["les", "linearized"])
@pytest.mark.parametrize("nx", [32, 128, 192])
def test_flux_tile_without_its_block(cf, nx, what):
    ends = []
    for tiles in ((3, 4, 8, 4), (3, 8, 8, 4), "own"):
        f = flow_of(cf, nx)
        f.set_tiles(f.tiles() if tiles == "own" else tiles)
        ends.append(steps(f, what))
        f.timestep(1)
        f.close()
    for e in ends[1:]:
        for a, b in zip(ends[0], e):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", [0, 1])
def test_tuned_les_context_steps(cf, prec):
    f = flow_of(cf, 192, prec=prec)
    f.set_les(1)
    for _ in range(4):
        f.autotune(1)
        assert f.tiles()[1] in (2, 4)
    f.timestep(2)
    f.set_les(0)
    f.timestep(2)
    assert f.status() == 0
    f.close()


@pytest.mark.parametrize("what", ["les", "linearized"])
def test_members_of_a_tuned_ensemble(cf, what):
    """Members step alone after the ensemble tuned them (twins take the first one's tiles)."""
    m = [flow_of(cf, 48) for _ in range(2)]
    m[0].set_les(1)      # keeps the ensemble off the batched layout
    ens = cf.Ensemble(m, autotune=True)
    ens.timestep(1)
    ens.synchronize()
    ens.close()
    for f in m:
        steps(f, what)
        f.close()
