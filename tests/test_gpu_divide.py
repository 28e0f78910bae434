"""The quotients of normalisations (divide_by_sum and divide_message in
csrc/bp_device.cuh) against IEEE fp32 division on the host, bit for bit:
zeros of both signs, subnormals, values whose quotients round in the subnormal
range or tie there, sums that are tiny, huge, infinite, zero or negative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _operands(S, seed, n=60_000):
    """[n, S] fp32 values of mixed kinds, rows of one kind and of several."""
    rng = np.random.default_rng(seed)
    u = rng.integers(0, 1 << 32, (n, S), dtype=np.uint32)
    kinds = [
        (u & 0x007FFFFF),                                   # subnormal
        (u & 0x03FFFFFF),                                   # near the subnormal border
        (u & 0x007FFFFF) | 0x3F000000,                      # [0.5, 1)
        (u % 0x7F000000),                                   # any magnitude, sum mostly finite
        np.zeros_like(u),
        (u & 0x000000FF),                                   # a few units of the smallest subnormal
        ((u & 0xFF) << 15) | 0x3F800000,                    # short mantissas: exact quotients and ties
        (u & 0x007FFFFF) | 0x7E800000,                      # sums that overflow to inf
    ]
    k = rng.integers(0, len(kinds), (n, S))
    rows = rng.random(n) < 0.5
    k[rows] = k[rows, :1]
    x = np.choose(k, kinds).astype(np.uint32)
    x ^= np.where(rng.random((n, S)) < 0.02, np.uint32(0x80000000), np.uint32(0))
    return x.view(F)


def _normalised(x):
    """The reference's order: the sum from 0 in state order, a sum <= 0 is 1."""
    s = np.zeros(len(x), F)
    with np.errstate(all="ignore"):
        for i in range(x.shape[1]):
            s = (s + x[:, i]).astype(F)
        s = np.where(s <= 0, F(1), s)
        return (x / s[:, None]).astype(F)


def _same_bits(got, want):
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])


@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 8, 10])
def test_belief_quotients(bp, synth, S):
    from belief_propagation_b200.engine import BPGraph
    b = _operands(S, seed=S)
    e = np.zeros(0, np.uint32)
    net = synth.Network(np.full(len(b), S, np.uint32), b, np.zeros(len(b), np.uint8), e, e, np.zeros((0, S, S), F))
    g = BPGraph.from_network(net)
    try:
        g.loopy(0.0, 1, delta="f64")
        _same_bits(g.beliefs(), _normalised(b))
    finally:
        g.close()


@pytest.mark.parametrize("S", [2, 3, 4, 7, 8])
def test_message_quotients(bp, synth, S):
    """Messages of a one-hot belief: the table's first column, normalised."""
    from belief_propagation_b200.engine import BPGraph
    x = _operands(S, seed=50 + S, n=20_000)
    x = np.where(np.isfinite(x), x, F(1)) + F(0)            # 0 + (-0) = +0, as the partial sums start
    joint = np.zeros((len(x), S, S), F)
    joint[:, :, 0] = x
    b = np.zeros((2, S), F)
    b[:, 0] = 1
    src, dst = np.zeros(len(x), np.uint32), np.ones(len(x), np.uint32)
    net = synth.Network(np.full(2, S, np.uint32), b, np.zeros(2, np.uint8), src, dst, joint)
    g = BPGraph.from_network(net)
    try:
        g.latest_slot = 1
        g.init_messages()
        _same_bits(g.messages(1), _normalised(x))
    finally:
        g.close()
