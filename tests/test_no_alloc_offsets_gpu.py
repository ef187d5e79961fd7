"""The allocation-free step on buffers that start at any element: the kernels of
16-byte accesses do not take them, the generic one does."""
import ctypes as C

import numpy as np
import pytest

from ic_helpers import smooth_noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,prec", [(1, 1 << 20, "fp64"), (2, 1024, "fp32c"), (2, 1500, "fp32c"), (2, 320, "fp64"),
                                      (3, 64, "fp32c"), (3, 64, "fp64")])
def test_buffers_off_by_one_element(d, n, prec):
    torch = pytest.importorskip("torch")
    import coolbubble_b200 as cb
    from coolbubble_b200 import _lib as L
    p = cb.make_params(d, n, n / 8.0, 4.0, 0.0125, precision=prec, memorysave=1)
    dt = torch.float64 if prec == "fp64" else torch.float32
    N = n ** d
    rng = np.random.default_rng(7)
    start = [0.4 + 0.1 * rng.standard_normal(N), 0.05 * rng.standard_normal(N)]
    got = []
    for off in (0, 1):
        bufs = [torch.zeros(N + 1, dtype=dt, device="cuda")[off:off + N] for _ in range(4)]
        for b, a in zip(bufs, start):
            b.copy_(torch.tensor(a, dtype=dt))
        torch.cuda.synchronize()
        out = L.cb_sums()
        L.check(L.lib.cb_step_static_noalloc(C.byref(p), *[b.data_ptr() for b in bufs], 0.0, C.byref(out)))
        got.append((bufs[2].cpu().numpy(), bufs[3].cpu().numpy(), out.asdict()))
    (phi, pi, a), (phi1, pi1, b) = got
    np.testing.assert_array_equal(phi, phi1)
    np.testing.assert_array_equal(pi, pi1)
    # the same terms in another order: N adds in double, or float terms compensated per thread
    tol = N * 2.0 ** -53 + (2.0 ** -20 if prec == "fp32c" else 0.0)
    for key in ("etot", "ekin", "egrad", "epot", "etot_var"):
        assert abs(a[key] - b[key]) <= tol * abs(a[key]), key
