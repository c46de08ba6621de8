"""Dependent launches: the steps of one timestep call overlap a kernel's start
with the end of the one before it, the same steps taken routine by routine do
not.  Every kernel has to see what its predecessors wrote (with an adaptive
time step the new dt as well), so both end in the same state, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny,nz,steps", [(32, 33, 32, 200), (48, 40, 24, 100), (64, 65, 64, 60), (128, 129, 96, 15)])
def test_steps_equal_their_routines(cf, nx, ny, nz, steps, prec):
    ends = []
    for chained in (True, False):
        f = cf.ChannelFlow(cf.Grid(nx, ny, nz, stretch=1.5), re=2500.0, dt=1e-3, dt_flag=1, cfl_max=0.4,
                           precision=prec)
        f.define_initial_field(10, seed=12, ampl=5e-2)
        if chained:
            f.timestep(steps)
        else:
            for s in range(1, steps + 1):
                f.boundary()
                for rk in (1, 2, 3):
                    f.nonlinear(s, rk)
                    f.rhs_solve(s, rk)
        sc = f.scalars()
        ends.append(list(f.download_state()) + [np.array([sc["dt"], sc["p_grad"], sc["cfl_max"]]), sc["d_um_dy"]])
        assert f.status() == 0
        f.close()
    assert ends[0][3][0] != 1e-3
    for a, b in zip(*ends):
        np.testing.assert_array_equal(a, b)
