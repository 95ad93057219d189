"""The marching kernels' chunk length follows the grid's size (march_chunk in
engine.cuh): the exact engine stays bit for bit with the oracle on grids whose
chunks are the shortest, uneven, and longer than an axis."""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import State
from lare3d_b200.grid import grid

pytestmark = pytest.mark.gpu
STATE = ("rho", "energy", "vx", "vy", "vz", "bx", "by", "bz")


@pytest.mark.parametrize("n", [(4, 4, 4), (5, 9, 33), (34, 6, 5), (61, 37, 29)])
def test_every_chunk_length_keeps_the_exact_state(built, n):
    from lare3d_b200 import gpu
    from oracle import oracle
    d0 = decks.orszag_tang(8, j_max=10.0, eta0=1.0e-3)
    st = State.zeros(*n)
    rng = np.random.default_rng(sum(n))
    for k in STATE:
        lo, hi = (0.5, 1.5) if k in ("rho", "energy") else (-0.3, 0.3)
        st[k][...] = rng.uniform(lo, hi, st[k].shape)
    d = decks.Deck("chunks", d0.params, *n, grid(*n, (0, 1.1), (0, 0.9), (0, 1.6)), st, nsteps=3)
    g, r = gpu.simulation(d, precision=gpu.EXACT64), oracle.simulation(d)
    for s in (g, r):
        s.start(d.state)
        for step in (1, 2, 3):
            s.step(step)
    for f in STATE:
        assert np.array_equal(g.get_field(f), r.get_field(f)), f
    g.close()
