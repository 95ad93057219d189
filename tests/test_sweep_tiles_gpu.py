"""The fused remap sweeps in the FP64 product build and in FP32, whose tiles,
limiters and start remainders are not the exact engine's, on the smallest and
on uneven grids: periodic, with walls, and with open sides, against the oracle.

A step rounds about a thousand operations behind a value, differences of
neighbouring values make up to eight times of it, and the limiters' branches are
continuous: three steps stay within 24,000 half ulps of a field's largest value.
"""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import BC_OPEN, BC_PERIODIC, BC_USER, State
from lare3d_b200.grid import grid

pytestmark = pytest.mark.gpu
STATE = ("rho", "energy", "vx", "vy", "vz", "bx", "by", "bz")


def deck(n, bc):
    sides = {f"{a}bc_{s}": bc for a in "xyz" for s in ("min", "max")}
    p = decks.default_params(gamma=5 / 3, visc1=0.1, visc2=0.5, dt_multiplier=0.8, resistive_mhd=1,
                             eta_background=1.0e-3, eta0=0.0, j_max=1.0e10, **sides)
    st = State.zeros(*n)
    rng = np.random.default_rng(sum(n) + bc)
    for k in STATE:
        lo, hi = (0.8, 1.2) if k in ("rho", "energy") else (-0.2, 0.2)
        st[k][...] = rng.uniform(lo, hi, st[k].shape)
    return decks.Deck("tiles", p, *n, grid(*n, (0, 1.1), (0, 0.9), (0, 1.6), bcs=(bc, bc, bc)), st, nsteps=3)


@pytest.mark.parametrize("precision,tol", [(64, 24e3 * 2.0 ** -53), (32, 24e3 * 2.0 ** -24)])
@pytest.mark.parametrize("bc", [BC_PERIODIC, BC_USER, BC_OPEN])
@pytest.mark.parametrize("n", [(4, 4, 4), (5, 9, 33), (29, 8, 7), (31, 7, 9), (34, 6, 5), (61, 37, 29)])
def test_three_steps_against_the_oracle(built, n, bc, precision, tol):
    from lare3d_b200 import gpu
    from oracle import oracle
    d = deck(n, bc)
    g, r = gpu.simulation(d, precision=precision), oracle.simulation(d)
    for s in (g, r):
        s.start(d.state)
        for step in (1, 2, 3):
            s.step(step)
    for f in STATE:
        a, b = g.get_field(f), r.get_field(f)
        assert np.isfinite(b).all()
        assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b)), f
    g.close()
