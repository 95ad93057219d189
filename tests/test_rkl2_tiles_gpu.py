"""The RKL2 stage kernel at the edges of its tiles (31 x 8 columns, chunks of
z down to 4 planes, the last stage writing the energy in place): conduct_heat
against the oracle at relative 1e-12, the bar of conduction's powers."""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import BC_PERIODIC, BC_USER, State
from lare3d_b200.grid import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(4, 4, 4), (31, 8, 5), (32, 9, 33), (63, 7, 17)])
@pytest.mark.parametrize("stages", [2, 3, 7])
def test_stage_tiles_against_the_oracle(built, n, stages):
    from lare3d_b200 import gpu
    from oracle import oracle
    p = decks.default_params(conduction=1, heat_flux_limiter=1, flux_limiter=0.1, kappa_0=1.0e-3,
                             kappa_perp_ratio=1.0e-3, zbc_min=BC_USER, zbc_max=BC_USER)
    st = State.zeros(*n)
    rng = np.random.default_rng(sum(n))
    for k in ("bx", "by", "bz"):
        st[k][...] = rng.uniform(-1.0, 1.0, st[k].shape)
    st["rho"][...] = rng.uniform(0.5, 2.0, st["rho"].shape)
    st["energy"][...] = rng.uniform(1.0, 4.0, st["energy"].shape)
    m = grid(*n, (0, 1.0), (0, 0.8), (0, 1.3), bcs=(BC_PERIODIC, BC_PERIODIC, BC_USER))
    d = decks.Deck("tiles", p, *n, m, st, nsteps=1)
    r = oracle.simulation(d)
    r.start(d.state)
    g = gpu.simulation(d, precision=gpu.FP64)
    g.start(d.state)
    dt = 1.0e-9
    while g.conduction_stages(dt) < stages:
        dt *= 1.25
    s = g.conduct_heat(dt)
    assert s >= stages and r.conduct_heat(dt) == s
    a, b = g.get_field("energy"), r.get_field("energy")
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    ta, tb = g.get_field("temperature"), r.get_field("temperature")
    assert np.max(np.abs(ta - tb)) <= 1e-12 * np.max(np.abs(tb))
    g.close()
