"""k_rhs_rows, the substep kernel with a thread per row: small grids take it
for every wavenumber (CHANFLOW_RHS_ROWS=0 keeps k_rhs2 there, =1 forces it),
all grids for the mean mode and the FP64 list.  One rhs_solve per substep
against the oracle at column heights around the block sizes (ny+1 of 6, 31,
32, 33, 64, 65 rows up to 256, the largest), with wall values on every
component.

The bars are the per-routine ones of test_gpu_parity.py (relative L2 1e-12 in
FP64 and 1e-5 in mixed precision, ten times that for the pressure; p_grad
1e-10 and 1e-6; d_um_dy 1e-12 and 1e-9).  They were set for 33 rows without
wall values; the rounding of taller columns, divided by dt and the wall
spacing, reaches the pressure beyond them on every path, so there the first
solver (CHANFLOW_RHS_V1) sets the bar: no further from the oracle than twice
its distance."""
import os

import numpy as np
import pytest

from test_gpu_parity import make, rel

pytestmark = pytest.mark.gpu


def solve(cf, orc, ny, prec, env):
    """Distances from the oracle of data1, data2, data4, p_grad and d_um_dy in each substep."""
    os.environ.update(env)
    try:
        grid, flow, o = make(cf, orc, 16, ny, 16, prec=prec)
    finally:
        for k in env:
            del os.environ[k]
    rng = np.random.default_rng(ny)
    o.init_field(10, seed=6, ampl=5e-2)
    top, bot = (1e-3 * (rng.standard_normal((16, 9, 3)) + 1j * rng.standard_normal((16, 9, 3))) for _ in range(2))
    o.cbc_top[...] = top
    o.cbc_bot[...] = bot
    out = []
    for rk in (1, 2, 3):
        o.set_step(1, rk)
        o.nonlinear()
        t, dt, pg = o.scalars()
        flow.upload_state(o.data1.copy(), o.data2.copy(), o.data4.copy())
        flow.set_scalars(t, dt, pg, o.d_um_dy.copy())
        flow.set_wall_bc(top, bot)
        o.rhs_solve()
        flow.rhs_solve(1, rk)
        sc = flow.scalars()
        out += [rel(a, b) for a, b in zip(flow.download_state(), (o.data1, o.data2, o.data4))]
        out += [abs(sc["p_grad"] / o.scalars()[2] - 1), rel(sc["d_um_dy"], o.d_um_dy)]
    flow.close()
    return np.array(out)


BARS = {0: (1e-12, 1e-12, 1e-11, 1e-10, 1e-12), 1: (1e-5, 1e-5, 1e-4, 1e-6, 1e-9)}


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("ny", [5, 30, 31, 32, 63, 64, 128, 200, 255])
def test_rhs_solve_rows(cf, orc, ny, prec):
    bar = np.maximum(np.tile(BARS[prec], 3), 2 * solve(cf, orc, ny, prec, {"CHANFLOW_RHS_V1": "1"}))
    for rows in ("0", "1"):
        got = solve(cf, orc, ny, prec, {"CHANFLOW_RHS_ROWS": rows})
        assert np.all(got <= bar), (rows, got, bar)
