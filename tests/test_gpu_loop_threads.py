"""Graphs of one state count, solved side by side by two host threads: the
one-launch loop takes shared memory by the graph (csrc/flood_loop.cuh), and
what one thread's graph takes is no concern of the other's launch."""
import threading

import numpy as np
import pytest

from test_kernel_source import _body, _code

ROUNDS = 1500


def test_no_launch_sets_a_limit_that_graphs_share():
    """A kernel's shared-memory limit belongs to the process.  The loop's is
    set while a graph is planned, to the device's own, and by no launch."""
    code = _code("loopy.cu")
    assert "cudaFuncSetAttribute" not in _body(code, r"static int launch_loop\(")
    plan = _body(code, r"static int loop_plan_of\(")
    limit = plan[plan.index("cudaFuncAttributeMaxDynamicSharedMemorySize"):]
    assert "smem" not in limit[len("cudaFuncAttributeMaxDynamicSharedMemorySize"):limit.index(";")]


@pytest.mark.gpu
@pytest.mark.parametrize("delta", ["f64", "serial"])
def test_two_threads_with_different_graphs(bp, synth, delta):
    from belief_propagation_b200.engine import BPGraph
    # 2,000 and 12 in-edges a tile: beyond 48 KB of shared memory, and little
    nets = [synth.random_loopy(512, 8000, 2, 0.1, seed=1), synth.random_loopy(500, 48, 2, 0.1, seed=2)]

    def solve(g, net):
        g.set_beliefs(net.beliefs)
        g.latest_slot = 1
        g.init_messages()
        g.loopy(0.0, 1, delta=delta)
        return g.beliefs()

    with BPGraph.from_network(nets[0]) as a, BPGraph.from_network(nets[1]) as b:
        alone = [solve(g, net) for g, net in zip((a, b), nets)]
        errors, wrong = [], []

        def work(g, net, ref):
            try:
                for _ in range(ROUNDS):
                    if not np.array_equal(solve(g, net), ref):
                        wrong.append(net.V)
            except Exception as e:
                errors.append(e)

        threads = [threading.Thread(target=work, args=x) for x in zip((a, b), nets, alone)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors and not wrong, (errors, wrong)
