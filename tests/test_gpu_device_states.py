"""Graphs whose arrays lie in device memory, with mixed state counts: the
state counts are scanned on the device (k_states_scan in csrc/engine.cu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _build(net, num_states, device):
    import torch
    from belief_propagation_b200.engine import BPGraph
    arrays = [net.src.astype(np.int32), net.dst.astype(np.int32), net.joint, num_states.astype(np.int32)]
    arrays = [torch.from_numpy(np.ascontiguousarray(x)) for x in arrays]
    if device:
        arrays = [x.cuda() for x in arrays]
    return BPGraph(net.V, arrays[0], arrays[1], arrays[2], num_states=arrays[3])


@pytest.mark.parametrize("V", [2, 31, 33, 255, 257, 5000])
def test_device_state_counts_build_the_host_graph(bp, synth, V):
    """The same tree from host and from device memory: equal shapes and, after
    both schedules, equal beliefs (the edge schedule walks the runs of equal
    state counts)."""
    net = synth.random_tree(V, (2, 3, 7), 0.05, seed=V)
    got = []
    for device in (False, True):
        g = _build(net, net.num_states, device)
        assert g.ms == net.num_states.max() and g.uniform == net.uniform_states
        out = []
        g.set_beliefs(net.beliefs)
        g.tree()
        out.append(g.beliefs())
        g.set_beliefs(net.beliefs)
        g.latest_slot = 1
        g.init_messages()
        g.loopy(0.0, 4, schedule="edge")
        out.append(g.beliefs())
        g.close()
        got.append(out)
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("bad", [0, 11, 1 << 30])
@pytest.mark.parametrize("device", [False, True])
def test_state_count_out_of_range_names_the_first_node(bp, synth, bad, device):
    from belief_propagation_b200.native import BPError
    net = synth.random_tree(700, (2, 3), 0.05, seed=1)
    ns = net.num_states.copy()
    ns[[299, 300, 650]] = bad
    with pytest.raises(BPError, match=f"node 299 has {bad} states"):
        _build(net, ns, device)
