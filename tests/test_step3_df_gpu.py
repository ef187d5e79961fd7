"""Plain steps of expanding 3-D runs on the marching kernel: against the
generic kernel, and many steps in one launch against one launch per step."""
import numpy as np
import pytest

from ic_helpers import bubbles, smooth_noise
from test_step_gpu import field_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,prec,alpha,L", [
    (128, "fp64", 0, 16.0),    # rows of whole warps in whole tiles
    (130, "fp64", 1, 13.0),    # vectors, the last tile over the end, dx^2 no power of two, gradient sums
    (129, "fp64", 0, 16.125),  # padded rows
    (251, "fp64", 0, 30.0),    # padded, several items per block; dx^2 has no two-operation division
    (260, "fp32c", 0, 32.5), (257, "fp32c", 1, 32.125), (288, "fp32c", 0, 36.0)])
def test_marching_kernel_equals_generic_kernel(n, prec, alpha, L, monkeypatch):
    import coolbubble_b200 as cb
    p = cb.make_params(3, n, L, 4.0, 0.1 * L / n, precision=prec, memorysave=1, expansion=1, mpl=10.0, alpha=alpha)
    phi0 = 0.4 + smooth_noise(3, n, 0.1, seed=3)
    pi0 = smooth_noise(3, n, 0.05, seed=4)
    many = cb.Bubble(p, phi0, pi0)
    monkeypatch.setenv("CB_STEP_PATH", "generic")
    generic = cb.Bubble(p, phi0, pi0)
    monkeypatch.undo()
    monkeypatch.setenv("CB_MULTI_STEP", "0")
    single = cb.Bubble(p, phi0, pi0)
    for k in (1, 4, 7):
        b, g = single.step(k, sums=True), generic.step(k, sums=True)
        monkeypatch.delenv("CB_MULTI_STEP")
        a = many.step(k, sums=True)
        monkeypatch.setenv("CB_MULTI_STEP", "0")
        assert a == b
    fa, fb, fg = many.fields(), single.fields(), generic.fields()
    for key in ("phi", "pi"):
        np.testing.assert_array_equal(fa[key], fb[key])
        # the box sums' order moves a by a unit in the last place of a sum
        assert field_err(fa[key], fg[key]) <= (1e-14 if prec == "fp64" else 12 * 2.0 ** -23), key
    for key in ("etot", "ekin", "egrad", "epot", "a", "H"):
        assert abs(a[key] - g[key]) <= (1e-12 if prec == "fp64" else 2.0 ** -21) * abs(g[key]), key
