"""Two tables and up to 8 states: the pull-form adjoint (k_u_bwd_pull2 in
csrc/unrolled.cu) against the scatter form and the fp64 torch reference, on
grids and on an irregular graph (nodes without out- or in-edges, repeated
edges, kinds that some nodes or all nodes lack)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(kind, seed):
    from belief_propagation_b200.unrolled import grid_tables
    rng = np.random.default_rng(seed)
    if kind == "grid":
        side = 19
        src, dst, tab = grid_tables(side)
        return side * side, src, dst, (tab | rng.integers(0, 2, len(tab) // 2).repeat(2)).astype(np.uint8)
    V, E = 300, 900
    src, dst = rng.integers(0, 200, E).astype(np.uint32), rng.integers(40, 260, E).astype(np.uint32)
    src[:20], dst[:20] = src[20:40], dst[20:40]
    tab = rng.integers(0, 2, E) | (0x80 * rng.integers(0, 2, E))
    if kind == "one kind":
        tab = np.full(E, 0x81)
    return V, src, dst, tab.astype(np.uint8)


@pytest.mark.parametrize("kind,S,T,ck", [("grid", 4, 7, 3), ("grid", 8, 6, 5), ("grid", 5, 1, 1), ("mixed", 1, 4, 2),
                                         ("mixed", 3, 5, 2), ("mixed", 6, 4, 4), ("mixed", 7, 3, 1),
                                         ("one kind", 2, 5, 2), ("one kind", 8, 3, 3)])
def test_two_table_pull_adjoint(bp, monkeypatch, kind, S, T, ck):
    import torch
    from belief_propagation_b200.unrolled import UnrolledBP, nll_loss, torch_unrolled
    V, src, dst, tab = _graph(kind, seed=10 * S + T)
    rng = np.random.default_rng(S)
    theta0, W0 = rng.normal(0, 1, (V, S)), rng.normal(0, 0.5, (2, S, S))
    labels = torch.tensor(rng.integers(0, S, V), device="cuda")
    res = []
    for pull in ("1", "0"):
        monkeypatch.setenv("BP_UBWD_PULL", pull)
        theta = torch.tensor(theta0, dtype=torch.float32, device="cuda", requires_grad=True)
        W = torch.tensor(W0, dtype=torch.float32, device="cuda", requires_grad=True)
        eng = UnrolledBP(V, src, dst, tab, S, T, checkpoint_every=ck, num_tables=2)
        lb = eng(theta, W)
        nll_loss(lb, labels).backward()
        res.append((lb.detach().cpu().numpy(), theta.grad.cpu().numpy(), W.grad.cpu().numpy()))
        eng.close()
    th64 = torch.tensor(theta0, dtype=torch.float64, device="cuda", requires_grad=True)
    W64 = torch.tensor(W0, dtype=torch.float64, device="cuda", requires_grad=True)
    torch.nn.functional.nll_loss(torch_unrolled(th64, W64, src, dst, tab, T), labels).backward()
    st, sw = th64.grad.abs().max().item(), W64.grad.abs().max().item()
    (lb1, gt1, gw1), (lb0, gt0, gw0) = res
    assert np.array_equal(lb1, lb0)
    for gt, gw in ((gt1, gw1), (gt0, gw0)):
        np.testing.assert_allclose(gt, th64.grad.cpu().numpy(), atol=1e-3 * st + 1e-7)
        np.testing.assert_allclose(gw, W64.grad.cpu().numpy(), rtol=1e-3, atol=1e-3 * sw + 1e-7)
    np.testing.assert_allclose(gt1, gt0, rtol=1e-4, atol=1e-5 * st + 1e-9)
    np.testing.assert_allclose(gw1, gw0, rtol=1e-4, atol=1e-5 * sw + 1e-9)
