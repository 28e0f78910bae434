"""A tuned batch with the f64 delta, below and above the work at which
bp_batch_autotune leaves the clusters: the tuned launch changes no network's
beliefs or iteration count (tolerance 0, so the delta's order decides nothing)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [12, 200])
def test_tuned_batch_changes_no_value(bp, synth, monkeypatch, tmp_path, count):
    from belief_propagation_b200.engine import BPBatch
    monkeypatch.setenv("BP_AUTOTUNE_CACHE", str(tmp_path / "tune"))
    nets = [synth.random_loopy(400, 1100 + 3 * (k % 5), 2, 0.1, seed=k) for k in range(count)]

    def solve(tune):
        b = BPBatch(nets)
        try:
            b.set_beliefs()
            if tune:
                b.autotune(tol=0.0, max_iterations=6)
                b.set_beliefs()
            b.loopy(tol=0.0, max_iterations=6)
            return b.beliefs(), b.results()["iterations"]
        finally:
            b.close()

    plain, tuned = solve(False), solve(True)
    np.testing.assert_array_equal(tuned[1], plain[1])
    for x, y in zip(tuned[0], plain[0]):
        np.testing.assert_array_equal(x, y)
