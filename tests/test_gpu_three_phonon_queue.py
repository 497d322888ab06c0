"""Three-phonon stage where a mode has more processes than its queue holds, so that the
queue is drained in whole rounds of the block and its rest moves to the front: more than
one drain, a rest of every size up to a round, and the fewest candidates."""
import pytest

import helpers as H
import oracle as O
import test_gpu_three_phonon_cells as cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,grid,most", [("layered", (3, 3, 3), 1024), ("random5", (3, 3, 3), 1024),
                                            ("random8", (2, 3, 3), 2048), ("diamond", (8, 8, 8), 2048),
                                            ("random7", (2, 2, 2), 0), ("diamond", (1, 1, 2), 0)])
def test_drains(cell, grid, most):
    n = O.Oracle(H.cached_solve(cell, grid)).np3()
    assert max(n[0].max(), n[1].max()) >= most
    cells.test_three_phonon_stage_matches_the_oracle(cell, grid)
