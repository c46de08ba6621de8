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


def test_training_batches_equal_separate_ones(cf):
    """The gradients of batches in a row, of changing sizes, against the same batches with a wait after each."""
    import torch
    rng = np.random.default_rng(2)
    x, t = (torch.from_numpy(rng.standard_normal((20000, n)).astype(np.float32)).cuda() for n in (10, 6))
    params = (0.1 * rng.standard_normal(9414)).astype(np.float32)
    idx = [torch.from_numpy(rng.integers(0, 20000, b).astype(np.int32)).cuda()
           for b in [20000] + [1, 127, 128, 129, 4096, 3000, 20000, 64] * 8]
    ends = []
    for wait in (False, True):
        m = cf.Mlp(params=params)
        for i in idx:
            m.accumulate_grad(x.data_ptr(), t.data_ptr(), i.data_ptr(), len(i))
            if wait:
                torch.cuda.synchronize()
        g, loss = m.grads()
        m.adam_step(1e-3)
        ends.append((g, np.float32(loss), m.get_params()))
        assert m.status() == 0
        m.close()
    for a, b in zip(*ends):
        np.testing.assert_array_equal(a, b)
