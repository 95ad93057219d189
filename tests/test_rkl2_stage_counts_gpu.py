"""RKL2 at forced stage counts (with two stages Y0, Y1 and the last stage's output
are all the energy array, with an even count the buffers end in another order),
with walls and with open sides, whose ghosts the stages carry, and the FP32
engine's stage tiles, whose rows have a length of their own.

The oracle's count follows from dt, so forced counts are compared where all
counts agree: RKL2 is of second order at any count, and dt is 2e-5 of the
explicit limit, so that counts differ by (2e-5)^3 times a few tens, below 1e-12,
the bar of conduction's powers, while a stage that read a value it should not
would show at the second order, 4e-10."""
import numpy as np
import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import BC_OPEN, BC_PERIODIC, BC_USER, State
from lare3d_b200.grid import grid

pytestmark = pytest.mark.gpu
SIZES = [(4, 4, 4), (31, 8, 5), (32, 9, 33), (63, 7, 17)]


def sims(n, zbc, precision):
    from lare3d_b200 import gpu
    from oracle import oracle
    p = decks.default_params(conduction=1, heat_flux_limiter=1, flux_limiter=0.1, kappa_0=1.0e-3,
                             kappa_perp_ratio=1.0e-3, zbc_min=zbc, zbc_max=zbc)
    st = State.zeros(*n)
    rng = np.random.default_rng(sum(n))
    for k in ("bx", "by", "bz"):
        st[k][...] = rng.uniform(-1.0, 1.0, st[k].shape)
    st["rho"][...] = rng.uniform(0.5, 2.0, st["rho"].shape)
    st["energy"][...] = rng.uniform(1.0, 4.0, st["energy"].shape)
    m = grid(*n, (0, 1.0), (0, 0.8), (0, 1.3), bcs=(BC_PERIODIC, BC_PERIODIC, zbc))
    d = decks.Deck("stages", p, *n, m, st, nsteps=1)
    g, r = gpu.simulation(d, precision=precision), oracle.simulation(d)
    for s in (g, r):
        s.start(d.state)
    dt = 1.0e-9
    while g.conduction_stages(dt) < 5:
        dt *= 1.1
    return g, r, dt / 2.5  # about the explicit limit


def check(g, r, tol):
    for f in ("energy", "temperature"):
        a, b = g.get_field(f), r.get_field(f)
        assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b)), f
    g.close()


@pytest.mark.parametrize("zbc", [BC_USER, BC_OPEN])
@pytest.mark.parametrize("stages", [2, 3, 4, 6])
@pytest.mark.parametrize("n", SIZES)
def test_forced_counts(built, n, stages, zbc):
    g, r, limit = sims(n, zbc, 64)
    before = g.get_field("energy")
    g.conduct_heat_stages(2e-5 * limit, stages)
    assert r.conduct_heat(2e-5 * limit) == 3
    # (the temperature is left as the last stage found it, which depends on the count)
    a, b = g.get_field("energy"), r.get_field("energy")
    assert np.max(np.abs(a - before)) > 1e-7 * np.max(np.abs(b))
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    g.close()


@pytest.mark.parametrize("ratio", [1.0, 12.0])
@pytest.mark.parametrize("n", SIZES)
def test_fp32_tiles(built, n, ratio):
    """About 40 roundings a stage and 7 stages: 300 half ulps, times 8 for the differences."""
    g, r, limit = sims(n, BC_USER, 32)
    s = g.conduct_heat(ratio * limit)
    assert s >= 3 and r.conduct_heat(ratio * limit) == s
    check(g, r, 2400 * 2.0 ** -24)
