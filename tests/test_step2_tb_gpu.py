"""Several steps per launch on static 1-D and 2-D lattices against one launch
per step: the same fields bit for bit; box sums on the bound of their adds."""
import numpy as np
import pytest

from ic_helpers import smooth_noise

pytestmark = pytest.mark.gpu

POSITIVE = ("etot", "ekin", "egrad", "epot", "etot_var", "ekin_var", "egrad_var", "epot_var", "avphi_var", "avphip_var")


@pytest.mark.parametrize("d,n,L", [
    (2, 5, 0.5),          # smaller than a tile's halo: coordinates wrap several times
    (2, 16, 2.0), (2, 32, 3.2), (2, 128, 16.0),   # a whole row on 8, 16 or 32 lanes
    (2, 64, 8.0), (2, 101, 12.625), (2, 250, 25.0),   # vectors, odd rows (site by site), double vectors only
    (2, 512, 32.0), (2, 1000, 100.0), (2, 1031, 103.1),   # several tiles, tiles over the end, more tiles than blocks
    (2, 288, 28.8), (2, 1024, 102.4),   # single steps with sums: the one-step kernels (1024: one strip a row)
    (2, 502, 30.0),       # dx^2 has no two-operation division: the compiler's divides
    (1, 3, 0.3), (1, 130, 16.25), (1, 4097, 409.7), (1, 1 << 18, 26214.4)])
@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
def test_multi_step_launches_equal_one_step_launches(d, n, L, prec, monkeypatch):
    import coolbubble_b200 as cb
    p = cb.make_params(d, n, L, 4.0, 0.1 * L / n, precision=prec, memorysave=1)
    phi0 = 0.4 + smooth_noise(d, n, 0.1, seed=3)
    pi0 = smooth_noise(d, n, 0.05, seed=4)
    many = cb.Bubble(p, phi0, pi0)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "1")
    single = cb.Bubble(p, phi0, pi0)
    monkeypatch.delenv("CB_TEMPORAL_BLOCK")
    N = n ** d
    # positive terms, each add rounded once: N 2^-53; float terms also rounded once
    # more by the compensated float accumulators of the one-step strip kernel
    tol = N * 2.0 ** -53 + (2.0 ** -23 if prec == "fp32c" else 2.0 ** -50)
    for steps, sums in ((1, True), (2, False), (7, True), (39, False), (40, True)):
        a, b = many.step(steps, sums=sums), single.step(steps, sums=sums)
        fa, fb = many.fields(), single.fields()
        np.testing.assert_array_equal(fa["phi"], fb["phi"])
        np.testing.assert_array_equal(fa["pi"], fb["pi"])
        if not sums:
            continue
        assert a["t"] == b["t"]
        for key in POSITIVE:
            assert abs(a[key] - b[key]) <= tol * abs(b[key]) + 1e-300, (steps, key)
        for key in ("avphi", "avphip"):
            assert abs(a[key] - b[key]) <= tol * (N * b[key + "_var"]) ** 0.5 + 1e-300, (steps, key)
    assert many.counters()[1] == single.counters()[1] == 89
    assert many.counters()[0] < 40 and single.counters()[0] == 89
