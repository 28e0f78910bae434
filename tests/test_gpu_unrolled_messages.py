"""The unrolled forward with stored messages (UMsgs in csrc/unrolled.cu)
against the form that recomputes each edge's message: the same values bit for
bit, forward and gradients, for one and several tables, one orientation only,
nodes without edges and segments of every length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(monkeypatch, form, V, src, dst, tab, S, T, ck, K, seed):
    import torch
    from belief_propagation_b200.unrolled import UnrolledBP, nll_loss
    monkeypatch.setenv("BP_UNROLLED_MSG", form)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    unary = torch.randn(V, S, generator=gen, device="cuda").requires_grad_()
    pair = (0.5 * torch.randn(K, S, S, generator=gen, device="cuda")).requires_grad_()
    labels = torch.randint(0, S, (V,), generator=gen, device="cuda")
    eng = UnrolledBP(V, src, dst, tab, states=S, iterations=T, checkpoint_every=ck, num_tables=K)
    lb = eng(unary, pair)
    nll_loss(lb, labels).backward()
    out = [x.detach().cpu().numpy() for x in (lb, unary.grad, pair.grad)]
    eng.close()
    return out


@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 8, 10])
@pytest.mark.parametrize("K,T,ck", [(1, 1, 5), (1, 7, 3), (2, 6, 5), (3, 5, 1)])
def test_stored_messages_equal_recomputed(bp, monkeypatch, S, K, T, ck):
    rng = np.random.default_rng(100 * S + 10 * K + T)
    V, E = 700, 2500                                       # some nodes without in- or out-edges
    src, dst = rng.integers(0, 600, E), rng.integers(50, V, E)
    tab = rng.integers(0, K, E) | (0x80 * rng.integers(0, 2, E))
    if K == 3:
        tab = tab & 0x7F                                   # one orientation only
    args = (V, src, dst, tab.astype(np.uint8), S, T, ck, K, S)
    for a, b in zip(_run(monkeypatch, "0", *args), _run(monkeypatch, "1", *args)):
        np.testing.assert_array_equal(a, b)
