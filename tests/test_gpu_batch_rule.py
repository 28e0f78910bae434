"""Which batches give their large networks a cluster each: the launch that a
batch is created with is not much slower than either fixed choice
(BP_BATCH_CLUSTER_EDGES), and its results are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _equal(synth, count, E, S):
    return [synth.random_loopy(E // 3, E, S, 0.1, seed=1)] * count


@pytest.mark.parametrize("name,clusters", [("few", True), ("many small", False), ("many of 8 states", True),
                                           ("many large of 2 states", False), ("uneven", True)])
def test_the_created_launch_is_near_the_better_one(bp, synth, monkeypatch, name, clusters):
    from belief_propagation_b200.engine import BPBatch
    nets = {"few": lambda: _equal(synth, 40, 3000, 3), "many small": lambda: _equal(synth, 1200, 1200, 2),
            "many of 8 states": lambda: _equal(synth, 300, 2400, 8),
            "many large of 2 states": lambda: _equal(synth, 600, 9600, 2),
            "uneven": lambda: synth.batch_of_networks(count=300, seed=2)}[name]()
    ms, bel = {}, {}
    for edges in (None, "0", "1024"):
        if edges is None:
            monkeypatch.delenv("BP_BATCH_CLUSTER_EDGES", raising=False)
        else:
            monkeypatch.setenv("BP_BATCH_CLUSTER_EDGES", edges)
        b = BPBatch(nets)
        try:
            t = []
            for _ in range(4):
                b.set_beliefs()
                t.append(b.loopy(tol=0.0, max_iterations=30)["elapsed_ms"])
            ms[edges], bel[edges] = min(t), b.beliefs()
        finally:
            b.close()
    # the choices lie 1.3 to 8 times apart here
    better, worse = ("1024", "0") if clusters else ("0", "1024")
    assert ms[better] < ms[worse]
    assert ms[None] < 1.15 * ms[better] + 0.02
    np.testing.assert_array_equal(bel[None], bel["0"])
    np.testing.assert_array_equal(bel["1024"], bel["0"])
