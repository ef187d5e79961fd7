"""Chains of plain steps replayed from a graph against plain launches, with the
launches of several steps turned off (they take such chains otherwise)."""
import numpy as np
import pytest

from ic_helpers import smooth_noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,prec,expansion", [
    (1, 4096, "fp64", 0), (2, 256, "fp32c", 0), (2, 512, "fp64", 0), (3, 96, "fp32c", 0), (3, 65, "fp64", 0),
    (3, 64, "fp32c", 1), (3, 64, "fp64", 1),
    (3, 128, "fp64", 1)])   # marches the planes in turn forwards and backwards: by the parity of the step
def test_replayed_chains_equal_plain_launches(d, n, prec, expansion, monkeypatch):
    """Fields, lines and time identical for chains that start from either buffer
    state and after an even or an odd number of steps."""
    import coolbubble_b200 as cb
    L = n / 8.0
    p = cb.make_params(d, n, L, 4.0, 0.1 * L / n, expansion=expansion, mpl=10.0, precision=prec, memorysave=1)
    start = 0.4 + smooth_noise(d, n, 0.1, seed=11), smooth_noise(d, n, 0.02, seed=12)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "1")   # static: one step per launch
    monkeypatch.setenv("CB_MULTI_STEP", "0")       # expanding: likewise
    graphed, plain = cb.Bubble(p, *start), cb.Bubble(p, *start)
    for steps in (17, 16, 32, 3, 20, 48, 1, 33):   # chains begin after 0, 17, 33, 65, 68, 88, ... steps
        monkeypatch.delenv("CB_STEP_GRAPHS", raising=False)
        graphed.step(steps, sums=False)
        monkeypatch.setenv("CB_STEP_GRAPHS", "0")
        plain.step(steps, sums=False)
        assert graphed.counters() == plain.counters()
        a, b = graphed.fields(local=False), plain.fields(local=False)
        for key in ("phi", "pi"):
            np.testing.assert_array_equal(a[key], b[key], err_msg=str(steps))
    assert graphed.step(1, sums=True) == plain.step(1, sums=True)
    assert plain.counters()[0] == plain.counters()[1]
