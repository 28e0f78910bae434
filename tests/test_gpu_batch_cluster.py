"""The batch's large networks, solved by a thread-block cluster each
(csrc/batch_cluster.cuh): against the oracle's beliefs and messages at fixed
iteration counts, and against the one-block solver, at sizes where blocks of a
cluster own few or no nodes, messages or tables do not fit shared memory, and
a hub's edges are one block's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(nets, monkeypatch, edges, **kw):
    from belief_propagation_b200.engine import BPBatch
    monkeypatch.setenv("BP_BATCH_CLUSTER_EDGES", str(edges))
    b = BPBatch(nets)
    try:
        b.set_beliefs()
        b.loopy(**kw)
        r = b.results()
        return [b.beliefs(k) for k in range(len(nets))], [b.messages(k) for k in range(len(nets))], r
    finally:
        b.close()


def _hub(synth, V, E, S, seed):
    net = synth.random_loopy(V, E, S, 0.1, seed=seed)
    dst = net.dst.copy()
    dst[: E // 2] = np.where(net.src[: E // 2] == 7, 8, 7)   # one node takes half of the edges
    return synth.Network(net.num_states, net.beliefs, net.observed, net.src, dst, net.joint, name="hub")


@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 8, 10])
def test_cluster_solver_gives_the_oracle_results(bp, synth, restatement, O, monkeypatch, S):
    nets = [synth.random_loopy(2, 1, S, 0.1, seed=1), synth.random_loopy(9, 40, S, 0.1, seed=2),
            synth.random_loopy(257, 1100, S, 0.1, seed=3), synth.random_loopy(3001, 17003, S, 0.1, seed=4),
            _hub(synth, 1500, 9000, S, seed=5), synth.random_loopy(600, 17000, S, 0.1, seed=6)]
    its = 7
    bel, msg, r = _solve(nets, monkeypatch, 1, tol=0.0, max_iterations=its)
    for k, net in enumerate(nets):
        ora = restatement.loopy(O.OracleGraph(net), 0.0, its)
        np.testing.assert_array_equal(bel[k], ora["beliefs"][:, :S])
        latest = ora["prev_arr"] if its % 2 == 0 else ora["cur_arr"]
        np.testing.assert_array_equal(msg[k], latest[:, :S])
        assert r["iterations"][k] == ora["ret"] and r["executed"][k] == ora["executed"]


def test_cluster_and_block_solver_agree_with_early_exits(bp, synth, monkeypatch):
    nets = synth.batch_of_networks(count=48, v_range=(32, 1500), seed=9)
    kw = dict(tol=1e-3, max_iterations=120)
    a = _solve(nets, monkeypatch, 0, **kw)
    b = _solve(nets, monkeypatch, 600, **kw)
    for k in range(len(nets)):
        np.testing.assert_array_equal(a[0][k], b[0][k])
        np.testing.assert_array_equal(a[1][k], b[1][k])
    for f in ("iterations", "executed", "converged"):
        np.testing.assert_array_equal(a[2][f], b[2][f])
    # the same terms summed in f64 in another order
    np.testing.assert_allclose(a[2]["delta"], b[2]["delta"], rtol=1e-6)


def test_second_solve_from_kept_messages(bp, synth, monkeypatch):
    """Without a new init a solve goes on from the messages the last one
    left (both arrays go back to memory)."""
    from belief_propagation_b200.engine import BPBatch
    nets = synth.batch_of_networks(count=6, v_range=(200, 900), seed=3)
    got = []
    for edges in (0, 1):
        monkeypatch.setenv("BP_BATCH_CLUSTER_EDGES", str(edges))
        b = BPBatch(nets)
        b.set_beliefs()
        b.loopy(tol=0.0, max_iterations=3)
        b.loopy(tol=0.0, max_iterations=2, init=False)
        b.set_beliefs()
        b.loopy(tol=0.0, max_iterations=1, init=False)
        got.append((b.beliefs(), b.messages()))
        b.close()
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
