"""Serial fp32 sums of 7M terms (csrc/serial_grid.cuh): so long a sum may drift
from the f64 prefix by half of it, and its slices guess the prefix's own binade
and the nearer neighbour.
The one-launch loop's deltas against a launch per iteration, whose sums one
block forms; the edge schedule's against the oracle."""
import numpy as np
import pytest

from test_gpu_loopy import assert_same, gpu_loopy

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(synth):
    V, E, S = 150000, 3500000, 2
    rng = np.random.default_rng(11)
    src = np.sort(rng.integers(0, V, E)).astype(np.uint32)
    dst = ((src + rng.integers(1, V, E)) % V).astype(np.uint32)
    j = rng.random((E, S, S), dtype=np.float32)
    j /= j.sum(2, keepdims=True)
    b = rng.dirichlet(np.ones(S), V).astype(np.float32)
    return synth.Network(np.full(V, S, np.uint32), b, np.zeros(V, np.uint8), src, dst, j, name="long")


def test_node_schedule(bp, net, monkeypatch):
    # a tolerance of 1 is far below the sums' rounding bounds: every check
    # forms its sum
    one = gpu_loopy(bp, net, 1.0, 8, delta="serial")
    monkeypatch.setenv("BP_FLOOD_FUSED", "0")
    launches = gpu_loopy(bp, net, 1.0, 8, delta="serial")
    np.testing.assert_array_equal(one["beliefs"], launches["beliefs"])
    for k in ("iterations", "delta", "previous_delta"):
        assert one[k] == launches[k], k
    assert one["serial_sums"] >= 4
    # a slice that no guess fits is added by one warp, which takes as long as the
    # one block's sums; guessed, the loop took a sixtieth of that
    assert 4 * one["elapsed_ms"] < launches["elapsed_ms"]


def test_edge_schedule(bp, net, restatement, O):
    for tol, its in ((0.0, 1), (1.0, 3)):
        ora = restatement.loopy(O.OracleGraph(net), tol, its, schedule="edge")
        assert_same(gpu_loopy(bp, net, tol, its, schedule="edge", delta="serial"), ora, 2)
