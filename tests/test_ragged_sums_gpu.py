"""Float lattices whose rows are padded: the sums take every site's term by
itself, as the generic kernel's did. Fields whose terms alternate between 1 and
2^-25 of it lose the small ones in any float sum of two sites."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,expansion,steps,line,alpha", [
    (65, 0, 1, True, 0), (66, 0, 1, True, 0), (67, 0, 1, True, 0)] + [   # reporting step, static
    (n, 1, steps, line, alpha) for n, steps, line in (
        (65, 1, True), (67, 1, True),                                # expanding
        (65, 1, False), (66, 1, False), (65, 3, False), (67, 3, False),   # Friedmann sums: a launch, several steps
        (257, 1, False), (259, 2, False))                            # marching kernel
    for alpha in (0, 1)])
def test_small_terms_beside_large_ones_are_summed(n, expansion, steps, line, alpha):
    import coolbubble_b200 as cb
    at = np.arange(n) % 4 < 2
    phi = np.broadcast_to(np.where(at, 1.0, 2.0 ** -25), (n, n, n)).reshape(-1)
    pi = np.broadcast_to(np.where(at, 1.0, 2.0 ** -13), (n, n, n)).reshape(-1)   # kinetic terms 2^-1 and 2^-27
    p = cb.make_params(3, n, n / 8.0, 4.0, 0.0, precision="fp32c", memorysave=1, expansion=expansion, mpl=10.0,
                       alpha=alpha)   # dt = 0: the fields stay what they are
    s = cb.Bubble(p, state=(phi, pi, dict(t=0.0, a=1.0, ap=0.0, H=0.0, ekin_half_prev=0.0, etot0=1.0)))
    s.step(steps, sums=line)
    got = s.sums()
    # a compensated float sum keeps 2 x 24 bits, a double 53; then a few roundings in double
    tol = 2.0 ** -40
    ek = math.fsum(0.5 * pi[:n] ** 2) / n
    assert abs(got["ekin_half_prev"] - ek) <= tol * ek
    if line:
        mean = math.fsum(phi[:n]) / n
        assert abs(got["avphi"] - mean) <= tol * mean
        assert abs(got["avphip_var"] * n ** 3 - math.fsum(pi[:n] ** 2) / n) <= tol
