"""bp_batch's block_threads governs every network, the ones large enough for a
cluster too, and the group reports describe the launch that runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(nets):
    from belief_propagation_b200.engine import BPBatch
    b = BPBatch(nets)
    b.set_beliefs()
    return b


def test_block_threads_governs_large_networks(bp, synth):
    """One network of 24,000 edges: a block takes several times as long as the
    eight of a cluster, and says so in the reports."""
    b = _batch([synth.random_loopy(4096, 24000, 8, 0.1, seed=1)])
    try:
        ms, bel, groups = {}, {}, {}
        for threads in (0, 256, 512, 0):
            for _ in range(2):
                b.set_beliefs()
                ms[threads] = b.loopy(tol=0.0, max_iterations=50, block_threads=threads)["elapsed_ms"]
            bel[threads], groups[threads] = b.beliefs(), b.groups()
        for threads in (256, 512):
            assert ms[threads] > 1.5 * ms[0]
            assert (groups[threads][0]["block"], groups[threads][0]["grid"]) == (threads, 1)
            np.testing.assert_array_equal(bel[threads], bel[0])
        assert (groups[0][0]["block"], groups[0][0]["grid"]) == (256, 8)
    finally:
        b.close()


def test_groups_report_both_launches(bp, synth):
    """Three networks by clusters and two by blocks; the serial delta takes a
    block for each."""
    nets = [synth.random_loopy(300, e, 3, 0.1, seed=e) for e in (1500, 1400, 1024, 1023, 60)]
    b = _batch(nets)
    try:
        assert b.groups() == [{"states": 3, "max_nodes": 0, "block": 256, "grid": 3 * 8 + 2}]
        b.loopy(tol=0.0, max_iterations=3, delta="serial")
        assert b.groups()[0]["grid"] == 5
        b.loopy(tol=0.0, max_iterations=3)
        assert b.groups()[0]["grid"] == 3 * 8 + 2
        b.loopy(tol=0.0, max_iterations=3, block_threads=128)
        assert b.groups() == [{"states": 3, "max_nodes": 0, "block": 128, "grid": 5}]
    finally:
        b.close()
