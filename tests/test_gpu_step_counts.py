"""Step counts near the 32-bit limit: the launches a call is split into."""
import pytest

from alpaca_b200 import api
from test_gpu_step_forms import box

pytestmark = pytest.mark.gpu

MOST = 2 ** 31 - 1


@pytest.mark.parametrize("n,parts", [((1, 1, 1), 4), ((37, 1, 1), 4), ((7, 7, 3), 2),
                                     ((37, 2, 2), 1)])
def test_tile_launches(cuda, n, parts):
    """Fused tile stages: three launches for as many steps as their items' 32-bit
    numbers hold (on 148 CTAs, one to an SM)."""
    c = box(3, n, True, 31)
    e = api.Engine(3, "fvchar", capacity_blocks=c.grid.nb, max_cases=1)
    e.add_case(c)
    e.set_path(4)
    most = (MOST - 148) // (3 * parts * c.grid.nb)
    assert [e.launches(k) for k in (1, most, most + 1)] == [3, 3, 6]
    assert e.launches(MOST) == 3 * -(-MOST // most)
    e.close()


@pytest.mark.parametrize("dim,n", [(1, (8, 1, 1)), (2, (2, 2, 1))])
def test_small_launches(cuda, dim, n):
    """Small 1D and 2D lists: a launch per 256 steps."""
    c = box(dim, n, True, 32)
    e = api.Engine(dim, "fvchar", capacity_blocks=c.grid.nb, max_cases=1)
    e.add_case(c)
    assert [e.launches(k) for k in (1, 256, 257, 512)] == [1, 1, 2, 2]
    assert e.launches(MOST) == 2 ** 23
    e.close()
