"""A context's device memory: 50 arrays of the engine's word and the 64-bit
staging of uploads and downloads.  What only some options need (conduction,
rke, partial ionisation) is allocated with them."""
import pytest

from lare3d_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,word", [(64, 8), (32, 4)])
def test_arrays_of_a_plain_context(built, precision, word):
    import torch
    from lare3d_b200 import gpu
    torch.cuda.init()
    d = decks.blast(8)
    gpu.simulation(d, precision=precision).close()  # loads the kernels
    n = 200
    d = decks.Deck("memory", d.params, n, n, n, decks.grid(n, n, n, (0, 1), (0, 1), (0, 1)), None, nsteps=1)
    free, _ = torch.cuda.mem_get_info()
    g = gpu.simulation(d, precision=precision)
    used = free - torch.cuda.mem_get_info()[0]
    points = 208 * 205 * 205
    assert used <= (50 * word + 8) * points * 1.05  # allocations are rounded up to 2 MiB
    g.close()
