"""Division of a Laplacian by dx^2 as two operations, fma(x, zh, x zl): correctly
rounded where the host accepts the divisor, and infinite for an infinite x."""
import ctypes as C
import random
from fractions import Fraction

import numpy as np
import pytest

from ic_helpers import smooth_noise


def pair(d):
    from coolbubble_b200 import _lib as L
    fn = L.lib["_ZN2cb15reciprocal_pairEdRdS0_"]   # cb::reciprocal_pair(double, double &, double &)
    fn.argtypes, fn.restype = [C.c_double, C.POINTER(C.c_double), C.POINTER(C.c_double)], C.c_bool
    zh, zl = C.c_double(), C.c_double()
    return (zh.value, zl.value) if fn(d, C.byref(zh), C.byref(zl)) else None


def quotient(x, zh, zl):
    return float(Fraction(x) * Fraction(zh) + Fraction(x * zl))   # float() of a Fraction rounds once, to nearest


def near_midpoints(d, most):
    """Integers X of 53 bits whose quotient by d's significand lies within most / (2 D) of a midpoint."""
    D = int(np.frexp(d)[0] * 2 ** 53)
    t = (D & -D).bit_length() - 1
    odd = D >> t
    out = []
    for e, lo, hi in ((53, D, 1 << 53), (54, 1 << 52, D)):
        for N in range(-most, most + 1):
            if N and odd > 1 and N % (1 << t) == 0:
                X = N * pow(2, -e, odd) % odd
                out += list(range(X + max(0, -(-(lo - X) // odd)) * odd, hi, odd))[:8]
    return out


def test_quotients_are_those_of_a_division():
    rng = random.Random(11)
    spacings = [0.1, 0.125, 0.0625, 0.2, 0.05, 0.15, 1 / 3] + [rng.uniform(1e-3, 4) for _ in range(300)]
    refused = 0
    for dx in spacings:
        d = dx * dx
        z = pair(d)
        if z is None:
            refused += 1
            continue
        xs = near_midpoints(d, 80) + [rng.uniform(-8, 8) for _ in range(20)] + [rng.randrange(1 << 52, 1 << 53) for _ in range(20)]
        for x in xs:
            assert quotient(float(x), *z) == float(x) / d, (dx, x)
    assert refused <= 24   # 3 % expected


@pytest.mark.parametrize("dx", [0.1, 0.125, 0.0625, 0.15, 0.2, 1 / 3])
def test_an_infinite_laplacian_has_an_infinite_quotient(dx):
    zh, zl = pair(dx * dx)
    for x in (np.inf, -np.inf):
        assert x * zh + x * zl == x


@pytest.mark.gpu
@pytest.mark.parametrize("d,n", [(1, 4097), (2, 64), (2, 250), (2, 1000)])
def test_refused_divisors_take_the_compilers_division(d, n, monkeypatch):
    """dx^2 without a pair: several steps per launch equal one per launch."""
    import coolbubble_b200 as cb
    L = n * 0.17
    assert pair((L / n) * (L / n)) is None
    p = cb.make_params(d, n, L, 4.0, 0.1 * L / n, memorysave=1)
    start = 0.4 + smooth_noise(d, n, 0.1, seed=3), smooth_noise(d, n, 0.05, seed=4)
    many = cb.Bubble(p, *start)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "1")
    single = cb.Bubble(p, *start)
    monkeypatch.undo()
    for steps, sums in ((40, True), (7, False)):
        a, b = many.step(steps, sums=sums), single.step(steps, sums=sums)
        fa, fb = many.fields(), single.fields()
        for key in ("phi", "pi"):
            np.testing.assert_array_equal(fa[key], fb[key])
        # the line's terms are positive, each add rounded once
        assert abs(a["etot"] - b["etot"]) <= (n ** d + 8) * 2.0 ** -53 * abs(b["etot"])


@pytest.mark.gpu
@pytest.mark.parametrize("d,n,dx,steps,expansion", [(2, 320, 0.1, 1, 0),    # several steps per launch, here one with sums
                                                    (3, 64, 0.1, 1, 0), (3, 64, 0.125, 1, 0),    # staged
                                                    (3, 64, 0.1, 2, 0),     # two-step pass
                                                    (3, 128, 0.1, 1, 1)])   # marching
def test_infinite_laplacians_step_as_by_division(d, n, dx, steps, expansion, monkeypatch):
    """A site whose neighbours are so large that its Laplacian is infinite: pi
    infinite there, and every site as in the kernel that divides."""
    import coolbubble_b200 as cb
    phi0, pi0 = smooth_noise(d, n, 0.1, seed=3).reshape((n,) * d), smooth_noise(d, n, 0.05, seed=4).reshape((n,) * d)
    at = (n // 2 + 1,) * d
    phi0[tuple(slice(a - 2, a + 3) for a in at)] = 0.0
    for ax in range(d):
        for s in (-1, 1):
            phi0[tuple(a + s * (i == ax) for i, a in enumerate(at))] = 0.8e308   # twice this is finite
    p = cb.make_params(d, n, n * dx, 4.0, 0.1 * dx, memorysave=1, expansion=expansion, mpl=10.0)
    start = phi0, pi0, dict(t=0.0, a=1.0, ap=0.0, H=0.0, ekin_half_prev=0.0, etot0=1.0)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "2")
    fast = cb.Bubble(p, state=start)
    monkeypatch.setenv("CB_STEP_PATH", "generic")
    by_division = cb.Bubble(p, state=start)
    monkeypatch.undo()
    for s in (fast, by_division):
        s.step(steps, sums=d == 2)
    a, b = fast.fields(), by_division.fields()
    if steps == 1:
        assert b["pi"].reshape((n,) * d)[at] == np.inf
    for key in ("phi", "pi"):
        np.testing.assert_array_equal(a[key], b[key])
