"""Creating an engine with two tables: the out-edges are put in kind order while
they are filled, so it takes what an engine with one table takes."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_tables_take_no_longer_to_create(bp):
    """512 x 512 grid.  Filled through the scatter form's slots and sorted node
    by node afterwards, two tables took 1.31 times one table's creation."""
    from belief_propagation_b200.unrolled import UnrolledBP, grid_tables
    side = 512
    src, dst, tab = grid_tables(side)
    two = (tab | np.random.default_rng(0).integers(0, 2, len(tab) // 2).repeat(2)).astype(np.uint8)
    times = [[], []]
    for _ in range(12):
        for k, t in enumerate((tab, two)):
            at = time.perf_counter()
            eng = UnrolledBP(side * side, src, dst, t, 5, 10, checkpoint_every=5, num_tables=k + 1)
            times[k].append(time.perf_counter() - at)
            eng.close()
    one, both = (float(np.median(t[2:])) for t in times)
    assert both < 1.15 * one, (one, both)
