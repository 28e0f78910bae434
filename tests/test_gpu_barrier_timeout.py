"""The one-launch loops' counter barrier gives up after a bounded wait: a block
is held back from every barrier (BP_DEBUG_BARRIER_SKIP) and the limit's base cut
to 50 ms (BP_DEBUG_WAIT_MS).  The call returns BP_ERR_TIMEOUT, nothing of it
stays in the barrier's counters, and the same graph then solves as it did
before.  One counter and two levels of them, both schedules, both deltas."""
import re

import numpy as np
import pytest

from test_kernel_source import _body, _code


def test_a_held_back_block_is_never_counted():
    """An arrival at a later barrier would stand for the missing one of an
    earlier: no wait need run out then, and the counters stay short."""
    code = _code("loopy.cu")
    barrier = _body(code, r"bool grid_barrier\(")
    arrive = re.search(r"if \(gb\.held\) \{\s*\} else if \(G <= kBarFlat\)", barrier)
    assert arrive and barrier.index("atomicAdd") > arrive.start()


@pytest.mark.gpu
@pytest.mark.parametrize("V,E,S,schedule,delta,check", [
    (12700, 25000, 2, "node", "f64", 1),       # 100 tiles: k_flood_fused, one counter
    (83000, 160000, 2, "node", "f64", 1),      # 649 tiles: two levels
    (83000, 160000, 2, "node", "f64", 4),
    (70000, 140000, 2, "node", "serial", 1),   # 547 tiles: k_flood_loop at the counter barrier
    (90000, 160000, 2, "node", "serial", 1),   # 704 tiles
    (20000, 50000, 3, "edge", "f64", 1),       # 196 blocks
    (20000, 50000, 3, "edge", "serial", 1),
    (200000, 400000, 2, "edge", "f64", 10),    # a full grid
])
def test_barrier_wait_runs_out_and_graph_stays_usable(bp, synth, monkeypatch, V, E, S, schedule, delta, check):
    from belief_propagation_b200.engine import BPGraph
    from belief_propagation_b200.native import BPError
    net = synth.random_loopy(V, E, S, 0.1, seed=V)
    zero = np.zeros((net.E, S), np.float32)

    def solve(g):
        g.set_beliefs(net.beliefs)
        g.set_messages(0, zero)
        g.set_messages(1, zero)
        g.latest_slot = 1
        g.init_messages()
        r = g.loopy(0.0, 20, check_every=check, schedule=schedule, delta=delta)
        return r["iterations"], r["delta"], g.beliefs()

    with BPGraph.from_network(net) as g:
        before = solve(g)
        for block in ("1", "0"):
            monkeypatch.setenv("BP_DEBUG_WAIT_MS", "50")
            monkeypatch.setenv("BP_DEBUG_BARRIER_SKIP", block)
            with pytest.raises(BPError) as err:
                solve(g)
            assert err.value.status == 8, err.value    # BP_ERR_TIMEOUT
            monkeypatch.delenv("BP_DEBUG_WAIT_MS")
            monkeypatch.delenv("BP_DEBUG_BARRIER_SKIP")
            after = solve(g)
            assert after[:2] == before[:2]
            np.testing.assert_array_equal(after[2], before[2])


@pytest.mark.gpu
@pytest.mark.parametrize("schedule,delta", [("edge", "f64"), ("edge", "serial"), ("node", "f64"), ("node", "serial")])
def test_barriers_wait_for_the_largest_node(bp, synth, monkeypatch, schedule, delta):
    """One node with a million in-edges: one thread multiplies their messages,
    27-43 ns each, while every other block waits.  The limit grows with the
    edges, so it does not run out even with a base of 1 ms."""
    from belief_propagation_b200.engine import BPGraph
    V, E, S = 1000, 1000000, 2
    rng = np.random.default_rng(5)
    j = rng.random((E, S, S), dtype=np.float32)
    net = synth.Network(np.full(V, S, np.uint32), np.full((V, S), 0.5, np.float32), np.zeros(V, np.uint8),
                        np.sort(rng.integers(1, V, E)).astype(np.uint32), np.zeros(E, np.uint32), j, name="hub")
    monkeypatch.setenv("BP_DEBUG_WAIT_MS", "1")
    with BPGraph.from_network(net) as g:
        g.latest_slot = 1
        g.init_messages()
        assert g.loopy(0.0, 2, schedule=schedule, delta=delta)["executed"] == 2
