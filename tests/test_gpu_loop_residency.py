"""The largest graphs of 5 states and more that run as one launch: every tile has a
resident block.  The route shows in the barrier's test hook, which a launch per
iteration does not have; the result is the same by either."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,S,mixed", [(75500, 6, False), (56500, 8, False), (56500, 7, False), (94000, 5, True),
                                       (75500, 8, True)])
def test_largest_one_launch_graphs(bp, synth, monkeypatch, V, S, mixed):
    from belief_propagation_b200.engine import BPGraph
    from belief_propagation_b200.native import BPError
    rng = np.random.default_rng(S)
    E = V
    src, dst = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    ns = np.where(rng.random(V) < 0.5, S, 2).astype(np.uint32) if mixed else np.full(V, S, np.uint32)
    live = np.arange(S) < ns[:, None]
    joint = rng.random((E, S, S), dtype=np.float32) * live[src][:, :, None] * live[dst][:, None, :]
    prior = rng.random((V, S), dtype=np.float32) * live
    with BPGraph(V, src, dst, joint, num_states=ns if mixed else None, uniform_states=0 if mixed else S) as g:
        got = []
        for fused in ("1", "0"):
            monkeypatch.setenv("BP_FLOOD_FUSED", fused)
            g.set_beliefs(prior)
            g.latest_slot = 1
            g.init_messages()
            g.loopy(0.0, 4, delta="f64")
            got.append(g.beliefs())
        np.testing.assert_array_equal(got[0], got[1])
        monkeypatch.setenv("BP_FLOOD_FUSED", "1")
        monkeypatch.setenv("BP_DEBUG_WAIT_MS", "50")
        monkeypatch.setenv("BP_DEBUG_BARRIER_SKIP", "1")
        with pytest.raises(BPError) as err:
            g.loopy(0.0, 4, delta="f64")
        assert err.value.status == 8   # BP_ERR_TIMEOUT
