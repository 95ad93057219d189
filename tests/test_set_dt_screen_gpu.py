"""set_dt's screening (lagran.cuh) on a grid whose blocks take several planes and
do not all run at once, so that cells are left out by the minima recorded
before them: dt of the exact engine equals the oracle's, also in units whose
lengths or densities lie at the edge of the 32-bit estimate's range or past it."""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import State
from lare3d_b200.grid import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,density,pressure", [
    (1.0, 1.0, 1.0),
    (1.0e-28, 1.0e25, 1.0),     # cells of 1e-30: around the least length that is judged
    (1.7e-43, 8.0e29, 2.0e-3),  # cells of 8.5e-46, which FP32 rounds to 1.4e-45
])
def test_dt_where_most_cells_are_left_out(built, length, density, pressure):
    from lare3d_b200 import gpu
    from oracle import oracle
    n = (200, 150, 60)
    d0 = decks.blast(8)
    st = State.zeros(*n)
    rng = np.random.default_rng(5)
    st["rho"][...] = density * rng.uniform(0.9, 1.1, st["rho"].shape)
    st["energy"][...] = pressure / density * rng.uniform(0.5, 1.5, st["rho"].shape)
    for k in ("bx", "by", "bz"):
        st[k][...] = 0.5 * np.sqrt(pressure) * rng.uniform(-1, 1, st[k].shape)
    d = decks.Deck("screen", d0.params, *n, grid(*n, (0, length), (0, length), (0, length)), st, nsteps=1)
    g, r = gpu.simulation(d, precision=gpu.EXACT64), oracle.simulation(d)
    for s in (g, r):
        s.start(d.state)
        s.lagrangian_step(1)
    assert np.isfinite(r.scalars().dt) and r.scalars().dt > 0
    assert g.scalars().dt == r.scalars().dt
    g.close()
