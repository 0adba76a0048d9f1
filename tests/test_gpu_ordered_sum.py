"""The ordered sum at the edges of its tiles (8 rows, 128 columns, a ring of 5) and of the chunk of row sums
that its last block holds (5200): the same bits as the oracle's serial chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 127), (8, 128), (9, 129), (16, 641), (17, 640), (5200, 2),
                                       (5201, 3), (10405, 15), (3, 5000)])
def test_tile_edges(sgpu_mod, oracle_mod, rows, cols):
    rng = np.random.default_rng(rows * 7919 + cols)
    v = rng.standard_normal((rows, cols)) * 10.0 ** rng.integers(-6, 6, (rows, cols))
    assert sgpu_mod.ordered_sum(v) == oracle_mod.ordered_sum(v)
