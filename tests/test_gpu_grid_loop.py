"""The one-launch loops of the node schedule against a launch per iteration:
tiles on both sides of the lines between the kernels (half the SMs, one tile
per SM, one counter or two levels in the grid barrier, the last size whose
tiles are all resident), and serial checks whose interval is narrowed.  Both
form every value and every sum in the same order, so nothing may differ."""
import numpy as np
import pytest

from test_gpu_loopy import gpu_loopy

pytestmark = pytest.mark.gpu


def _both(bp, net, monkeypatch, tol, its, **kw):
    one = gpu_loopy(bp, net, tol, its, **kw)
    monkeypatch.setenv("BP_FLOOD_FUSED", "0")
    return one, gpu_loopy(bp, net, tol, its, **kw)


def _assert_equal(a, b):
    np.testing.assert_array_equal(a["beliefs"], b["beliefs"])
    for k in ("iterations", "delta", "delta_f64"):
        assert a[k] == b[k], k


@pytest.mark.parametrize("tiles", [74, 75, 148, 149, 640, 641, 1776, 1777])
@pytest.mark.parametrize("S", [2, 3, 5, 7])
def test_f64_loops(bp, synth, monkeypatch, tiles, S):
    V = tiles * (256 if S == 3 else 128) - 127
    net = synth.random_loopy(V, V * 3 // 2, S, 0.1, seed=tiles + S)
    for check in (1, 4):
        _assert_equal(*_both(bp, net, monkeypatch, 1e-3, 18, check_every=check, delta="f64"))
        monkeypatch.delenv("BP_FLOOD_FUSED")


@pytest.mark.parametrize("V,S", [(20000, 2), (76000, 2), (40000, 3), (9000, 8)])
def test_serial_checks(bp, synth, monkeypatch, V, S):
    net = synth.random_loopy(V, 3 * V, S, 0.1, seed=V)
    for tol in (1e-3, 1.0):
        _assert_equal(*_both(bp, net, monkeypatch, tol, 40, delta="serial"))
        monkeypatch.delenv("BP_FLOOD_FUSED")
