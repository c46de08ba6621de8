"""Device arrays of callers that start at any float (4 bytes): the closure
network's features, targets and outputs at an odd offset give the bits of the
aligned arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shifted(a):
    """a's values in an array that starts one float past an allocation."""
    import torch
    b = torch.empty(a.numel() + 1, dtype=a.dtype, device=a.device)
    b[1:] = a.reshape(-1)
    assert b[1:].data_ptr() % 8 == 4
    return b[1:]


@pytest.mark.parametrize("n", [1, 127, 1000, 70000])
def test_network_arrays_at_an_odd_float(cf, n):
    import torch
    rng = np.random.default_rng(n)
    x, t = (torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32)).cuda() for k in (10, 6))
    idx = torch.from_numpy(rng.integers(0, n, 700).astype(np.int32)).cuda()
    net = cf.Mlp(params=(0.2 * rng.standard_normal(9414)).astype(np.float32))
    ends = []
    for move in (lambda a: a, shifted):
        xs, ts, y = move(x), move(t), move(torch.zeros((n, 6), device="cuda"))
        net.forward(xs.data_ptr(), y.data_ptr(), n)
        net.zero_grads()
        net.accumulate_grad(xs.data_ptr(), ts.data_ptr(), idx.data_ptr(), 700)
        g, loss = net.grads()
        ends.append((y.cpu().numpy().reshape(-1), g, np.float32(loss)))
    assert net.status() == 0
    assert ends[0][0].any() and ends[0][1].any()
    for a, b in zip(*ends):
        np.testing.assert_array_equal(a, b)
    net.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_les_features_at_an_odd_float(cf, prec):
    import torch
    f = cf.ChannelFlow(cf.Grid(32, 17, 32, stretch=1.5), re=3000.0, dt=0.004, precision=prec)
    f.define_initial_field(10, seed=4, ampl=5e-2)
    f.set_les(2, mlp=cf.Mlp(params=np.zeros(9414, np.float32)))
    n = (f.ny - 1) * f.grid.nz2 * f.grid.nx2 * 10
    a = torch.zeros(n, device="cuda")
    b = shifted(torch.zeros(n, device="cuda"))
    for out in (a, b):
        f.les_features(out.data_ptr())
        f.synchronize()
    assert a.cpu().numpy().any()
    np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    f.close()
