"""The edge schedule's one-launch loop (csrc/edge_loop.cuh) against the oracle:
grids of one block and of many, node 0's repeated normalisation over long runs
of equal state counts (where its orbit ends in a cycle), and every
state-count shape."""
import numpy as np
import pytest

from test_gpu_loopy import assert_same, gpu_loopy

pytestmark = pytest.mark.gpu


def _grouped_states(synth, V, E, choices, seed):
    """A graph whose nodes come in runs of equal state counts."""
    base = synth.random_loopy(V, E, 2, 0.1, seed=seed)
    rng = np.random.default_rng(seed)
    ns = np.sort(rng.choice(np.array(choices, np.uint32), size=V))
    S = int(max(choices))
    b = rng.random((V, S), dtype=np.float32) * (np.arange(S)[None] < ns[:, None])
    j = rng.random((E, S, S), dtype=np.float32)
    j *= np.arange(S)[None, :, None] < ns[base.src][:, None, None]
    j *= np.arange(S)[None, None, :] < ns[base.dst][:, None, None]
    return synth.Network(ns, b.astype(np.float32), base.observed, base.src, base.dst, j.astype(np.float32))


@pytest.mark.parametrize("delta", ["serial", "f64"])
@pytest.mark.parametrize("V,E,S", [(2, 1, 2), (255, 257, 3), (257, 1021, 10), (5001, 20003, 3), (40001, 80003, 2)])
def test_edge_loop_sizes(bp, synth, restatement, O, V, E, S, delta):
    net = synth.random_loopy(V, E, S, 0.1, seed=V)
    for check, its in ((1, 9), (10, 21)):
        ora = restatement.loopy(O.OracleGraph(net), 0.0, its, check_every=check, schedule="edge")
        gpu = gpu_loopy(bp, net, 0.0, its, check_every=check, schedule="edge", delta=delta)
        if delta == "serial":
            assert_same(gpu, ora, S)
        else:
            # tolerance 0 never stops: the same values without the serial sum
            np.testing.assert_array_equal(gpu["beliefs"][:, :S], ora["beliefs"][:, :S])
            assert gpu["iterations"] == ora["ret"]


@pytest.mark.parametrize("choices", [(2, 3), (3, 5, 8), (1, 4)])
def test_edge_loop_runs_of_equal_state_counts(bp, synth, restatement, O, choices):
    net = _grouped_states(synth, 3000, 9001, choices, seed=sum(choices))
    S = max(choices)
    ora = restatement.loopy(O.OracleGraph(net), 1e-3, 12, schedule="edge")
    assert_same(gpu_loopy(bp, net, 1e-3, 12, schedule="edge"), ora, S)
