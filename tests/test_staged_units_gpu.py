"""The planes per work unit of the staged passes on grids of three or more tiles
along z: orders 1 and 3 and orders 2 and 4 follow their own forms of the rule
(order 4 fast at 240 x 180 x 160 492 us per step with 8 planes, 502 with 6;
order 1 at 200^3 396 with 5, 418 with 2)."""
import pytest

from cases import case3d, product3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,N,exact,least,most", [
    ((240, 180, 160), 4, False, 8, 12), ((200, 200, 200), 1, True, 4, 8), ((200, 200, 200), 2, True, 4, 6)])
def test_units(cuda, shape, N, exact, least, most):
    p = product3d(case3d(shape=shape, N=N, nt=4, hetero=False), exact=exact)._build_plan()
    assert p.info()["path"] == "staged"
    assert least <= p.info()["staged_chunk"] <= most
