"""A tile copy that never arrives: the kernels' wait for it ends by itself, and
the context's calls then say so.  The wait is made to run out by a block that
waits on a barrier for which no copy was asked."""
import ctypes as C

import pytest

from lare3d_b200 import decks
from lare3d_b200.abi import LareError

pytestmark = pytest.mark.gpu


def lose_a_copy(sim):
    from lare3d_b200 import gpu
    f = gpu.library().lare_gpu_check_lost_copy
    f.argtypes = [C.c_void_p, C.POINTER(C.c_double)]
    t = (C.c_double * 2)()
    assert f(sim.ctx, t) == 0
    return t[0], t[1]


@pytest.mark.parametrize("precision", [64, 65, 32])
def test_every_call_that_waits_reports_it(built, precision):
    from lare3d_b200 import gpu
    d = decks.conduction(8)
    g = gpu.simulation(d, precision=precision)
    g.start(d.state)
    g.energy()
    first, later = lose_a_copy(g)
    assert 0.1 < first < 4.0   # about a second
    assert later < 0.02        # not waited for
    calls = [g.energy, g.download, g.scalars, lambda: g.get_field("rho"), lambda: g.conduct_heat(1e-9),
             lambda: g.conduction_stages(1e-9), lambda: g.step(1), lambda: g.run(1, 1)]
    for q, call in enumerate(calls + calls):  # the status stays
        with pytest.raises(LareError, match="copy") as e:
            call()
        assert e.value.code == -2, q
    g.close()


def test_a_later_status_does_not_replace_it(built):
    """An ionisation bracket that is empty raises LARE_EEOS, and does not hide a lost copy."""
    from lare3d_b200 import gpu
    d = decks.partially_ionised(8)
    g = gpu.simulation(d)
    g.start(d.state)
    lose_a_copy(g)
    e = g.b.lib.lare_gpu_set_field
    a = d.state["energy"].copy(order="F")
    a[...] = 0.0
    e.argtypes = [C.c_void_p, C.c_char_p, C.POINTER(C.c_double)]
    assert e(g.ctx, b"energy", a.ctypes.data_as(C.POINTER(C.c_double))) == 0
    for _ in range(2):
        with pytest.raises(LareError) as err:
            g.neutral_fraction()
        assert err.value.code == -2
    g.close()


def test_the_context_next_to_it_goes_on(built):
    """The GPU and other contexts stay usable."""
    from lare3d_b200 import gpu
    d = decks.blast(8)
    a, b = gpu.simulation(d), gpu.simulation(d)
    for s in (a, b):
        s.start(d.state)
    lose_a_copy(a)
    b.step(1)
    assert b.scalars().dt > 0
    for s in (a, b):
        s.close()
