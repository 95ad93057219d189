"""neutral_fraction visits the reference's bisection midpoints but evaluates
the ionisation balance only where the sign is not already known: the exact
engine's xi_n equals the oracle's full bisection bit for bit over cold, hot,
thin and dense cells, roots next to either end of the bracket among them."""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import EOS_ION, EOS_PI

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eos", [EOS_ION, EOS_PI])
@pytest.mark.parametrize("log_rho", [(-6.0, -2.0), (-2.0, 2.0), (2.0, 6.0)])
@pytest.mark.parametrize("log_t", [(-1.3, -0.3), (-0.3, 0.7), (0.7, 3.0)])
def test_xi_equals_the_full_bisection(built, eos, log_rho, log_t):
    from lare3d_b200 import gpu
    from oracle import oracle
    n = 16
    d = decks.partially_ionised(n, eos_number=eos, cowling=False)
    rng = np.random.default_rng(int(100 * log_rho[0] + 10 * log_t[0]) + 7000 + eos)
    shape = d.state["rho"].shape
    rho = np.asfortranarray(10.0 ** rng.uniform(*log_rho, shape))
    T = 10.0 ** rng.uniform(*log_t, shape)
    p = d.params
    c = {k: getattr(p, k) for k in ("f_bar", "t_bar", "r_bar", "tr")}
    with np.errstate(over="ignore", invalid="ignore"):
        xi = np.nan_to_num(decks.get_neutral(T, rho, c), nan=1.0)
    e = (T * (2.0 - xi) + (1.0 - xi) * p.ionise_pot * (p.gamma - 1.0)) / (p.gamma - 1.0)
    # some cells at the ends: all neutral, all ionised
    e.flat[::97] = 1.0e-3
    e.flat[::101] = 1.0e4
    out = []
    for prec in (gpu.EXACT64, None):
        s = gpu.simulation(d, precision=prec) if prec else oracle.simulation(d)
        s.set_field("rho", rho)
        s.set_field("energy", np.asfortranarray(e))
        s.neutral_fraction()
        out.append(s.get_field("xi_n"))
        s.close()
    a, b = out
    assert np.array_equal(a, b, equal_nan=True), np.abs(a - b).max()
