"""The named fields bx1, by1 and bz1 hold the magnetic field before the last
resistive sub-cycle (lagran.F90:1259-1261), and zeros where none has run: the
predictor's and the remap's sweeps leave them alone."""
import numpy as np
import pytest

from lare3d_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 65, 32])
def test_b_before_the_subcycle(built, precision):
    from lare3d_b200 import gpu
    d = decks.orszag_tang(12)
    g = gpu.simulation(d, precision=precision)
    g.start(d.state)
    for step in range(1, 8):  # more than the remap's six orders of axes
        before = {f: g.get_field(f) for f in ("bx", "by", "bz")}
        g.step(step)
        assert g.scalars().last_substeps == 1
        for q, f in enumerate(("bx", "by", "bz")):
            cells = [slice(1 if k == q else 0, None) for k in range(3)]  # from -1 along the face's axis
            assert np.array_equal(g.get_field(f + "1"), before[f][tuple(cells)]), (step, f)
    g.close()


def test_zeros_without_resistivity(built):
    from lare3d_b200 import gpu
    d = decks.blast(12)
    g = gpu.simulation(d)
    g.start(d.state)
    for step in (1, 2):
        g.step(step)
    for f in ("bx1", "by1", "bz1"):
        assert not g.get_field(f).any(), f
    g.close()
