"""Two leapfrog steps per pass on static 3-D lattices against one step per
pass: the same fields bit for bit, in float and double, for rows that are
whole warps and rows that are not, tiles that divide the lattice and tiles
that hang over its end."""
import numpy as np
import pytest

from ic_helpers import smooth_noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,prec", [
    (128, 16.0, "fp32c"), (132, 13.2, "fp32c"), (192, 24.0, "fp32c"), (200, 20.0, "fp32c"),
    (64, 8.0, "fp64"), (66, 6.6, "fp64"), (128, 12.8, "fp64"), (130, 16.25, "fp64")])
def test_two_step_pass_equals_one_step_passes(n, L, prec, monkeypatch):
    import coolbubble_b200 as cb
    p = cb.make_params(3, n, L, 4.0, 0.1 * L / n, precision=prec, memorysave=1)
    phi0 = 0.4 + smooth_noise(3, n, 0.1, seed=3)
    pi0 = smooth_noise(3, n, 0.05, seed=4)
    runs = []
    for steps in ("2", "1"):
        monkeypatch.setenv("CB_TEMPORAL_BLOCK", steps)
        runs.append(cb.Bubble(p, phi0, pi0))
    two, one = runs
    for k in (2, 7, 4):
        a, b = two.step(k, sums=k != 2), one.step(k, sums=k != 2)
        assert a == b
        fa, fb = two.fields(), one.fields()
        np.testing.assert_array_equal(fa["phi"], fb["phi"])
        np.testing.assert_array_equal(fa["pi"], fb["pi"])
    assert two.counters() == (1 + 4 + 3, 13) and one.counters() == (13, 13)


@pytest.mark.parametrize("dx", [0.1, 0.125])
def test_two_step_pass_of_128_vectors_a_row_in_double(dx, monkeypatch):
    """256^3 in double, rows whose shared offsets are constants of the kernel:
    dx^2 that divides in two operations and in one."""
    import coolbubble_b200 as cb
    n = 256
    rng = np.random.default_rng(5)
    start = 0.4 + 0.1 * rng.standard_normal(n ** 3), 0.05 * rng.standard_normal(n ** 3)
    p = cb.make_params(3, n, n * dx, 4.0, 0.1 * dx, precision="fp64", memorysave=1)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "2")
    two = cb.Bubble(p, *start)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "1")
    one = cb.Bubble(p, *start)
    for k in (2, 7):
        a, b = two.step(k, sums=k != 2), one.step(k, sums=k != 2)
        assert a == b
        fa, fb = two.fields(), one.fields()
        np.testing.assert_array_equal(fa["phi"], fb["phi"])
        np.testing.assert_array_equal(fa["pi"], fb["pi"])
    assert two.counters() == (1 + 4, 9) and one.counters() == (9, 9)
