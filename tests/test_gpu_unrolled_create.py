"""Creating an engine with two tables: the pull form's out-edges are put in kind
order while they are filled, so it takes no longer than the scatter form's."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pull_form_of_two_tables_takes_no_longer_to_create(bp, monkeypatch):
    """512 x 512 grid.  Filled through the scatter form's slots and sorted node
    by node afterwards, the pull form took 1.4 times as long."""
    from belief_propagation_b200.unrolled import UnrolledBP, grid_tables
    side = 512
    src, dst, tab = grid_tables(side)
    tab = (tab | np.random.default_rng(0).integers(0, 2, len(tab) // 2).repeat(2)).astype(np.uint8)
    times = {"1": [], "0": []}
    for _ in range(12):
        for pull, out in times.items():
            monkeypatch.setenv("BP_UBWD_PULL", pull)
            at = time.perf_counter()
            eng = UnrolledBP(side * side, src, dst, tab, 5, 10, checkpoint_every=5, num_tables=2)
            out.append(time.perf_counter() - at)
            eng.close()
    pull, scatter = (float(np.median(times[k][2:])) for k in "10")
    assert pull < 1.15 * scatter, (pull, scatter)
