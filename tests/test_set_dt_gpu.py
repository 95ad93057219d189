"""set_dt leaves out the cells whose limits lie above the minima recorded so
far (lagran.cuh): dt and dtr of the exact engine stay equal to the oracle's
where the sound speed, the flow or the resistivity limits the step, for
densities inside and outside the range that its 32-bit estimate can judge, and
where every cell has the same limit."""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import State
from lare3d_b200.grid import grid

pytestmark = pytest.mark.gpu


def _step(sim, state):
    sim.start(state)
    sim.step(1)
    return sim.scalars()


@pytest.mark.parametrize("density", [1.0, 1.0e-25, 1.0e-36, 1.0e34])
@pytest.mark.parametrize("speed,spread", [(0.3, 0.5), (30.0, 0.5), (0.0, 0.0)])
def test_dt_equals_the_oracles(built, density, speed, spread):
    from lare3d_b200 import gpu
    from oracle import oracle
    n = (69, 21, 43)  # two blocks across, the last chunk of planes ragged
    d0 = decks.orszag_tang(8, j_max=10.0, eta0=1.0e-3)
    st = State.zeros(*n)
    rng = np.random.default_rng(7)
    for k, scale in (("rho", density), ("energy", 1.0)):
        st[k][...] = scale * (1.0 + spread * rng.uniform(-1, 1, st[k].shape))
    for k in ("vx", "vy", "vz"):
        st[k][...] = speed * rng.uniform(-1, 1, st[k].shape)
    for k in ("bx", "by", "bz"):
        st[k][...] = 0.2 * np.sqrt(density) * spread * rng.uniform(-1, 1, st[k].shape)
    d = decks.Deck("limits", d0.params, *n, grid(*n, (0, 1.1), (0, 0.9), (0, 1.6)), st, nsteps=1)
    g, r = gpu.simulation(d, precision=gpu.EXACT64), oracle.simulation(d)
    sg, sr = [_step(s, d.state) for s in (g, r)]
    assert np.isfinite(sr.dt) and sr.dt > 0
    assert sg.dt == sr.dt and sg.dtr == sr.dtr
    g.close()
