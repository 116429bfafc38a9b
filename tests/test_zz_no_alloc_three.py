"""logo_best_move_noalloc with three cities, which have no pair of edges to
exchange: there is nothing to evaluate, so cities any distance apart are
answered (no move), while from four on the diagonal's limit holds."""
import numpy as np
import pytest

from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,want", [(3, 0), (4, 1)])
def test_cities_beyond_the_diagonal_limit(lg, n, want):
    torch = pytest.importorskip("torch")
    xy = np.array([[0, 0], [5.0e6, 0], [0, 5.0e6], [5.0e6, 5.0e6]], dtype=np.float32)[:n]
    assert _noalloc(lg, torch, xy, np.arange(n, dtype=np.uint32)) == ((0, 0, 0), want)
