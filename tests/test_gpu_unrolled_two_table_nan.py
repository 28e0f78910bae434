"""Two tables, a node whose state is NaN: its own messages are, and the gradient
of a table that none of its out-edges uses is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 3, 4, 5, 8])
def test_nan_stays_with_the_tables_its_edges_use(bp, S):
    import torch
    from belief_propagation_b200.unrolled import UnrolledBP, nll_loss
    V, E = 200, 700
    rng = np.random.default_rng(S)
    src, dst = rng.integers(2, V, E).astype(np.uint32), rng.integers(2, V, E).astype(np.uint32)
    tab = (rng.integers(0, 2, E) | (0x80 * rng.integers(0, 2, E))).astype(np.uint8)
    src[0], dst[0], tab[0] = 0, 1, 0    # the NaN node's only edge, to a node that sends nothing
    theta0, W0 = rng.normal(0, 1, (V, S)).astype(np.float32), rng.normal(0, 0.5, (2, S, S)).astype(np.float32)
    labels = torch.tensor(rng.integers(0, S, V), device="cuda")
    engine = UnrolledBP(V, src, dst, tab, S, 3, 2, 2)
    grads = []
    for bad in (False, True):
        theta0[0] = np.nan if bad else 0.1
        theta = torch.tensor(theta0, device="cuda", requires_grad=True)
        W = torch.tensor(W0, device="cuda", requires_grad=True)
        nll_loss(engine(theta, W), labels).backward()
        grads.append((theta.grad.cpu().numpy(), W.grad.cpu().numpy()))
    engine.close()
    (gu, gp), (nu, np_) = grads
    assert np.isfinite(gp).all() and np.isnan(np_[0]).all()
    np.testing.assert_array_equal(np_[1], gp[1])
    np.testing.assert_array_equal(nu[2:], gu[2:])
