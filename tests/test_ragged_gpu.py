"""3-D lattices whose rows are no whole number of 16-byte vectors: the run keeps
them padded (the pad holds the row's first sites again), the caller sees dense
fields. Staged and two-step kernels against the generic one and the oracle."""
import numpy as np
import pytest

from ic_helpers import bubbles, smooth_noise
from test_step_gpu import FIELD_TOL, _oracle_run, check_sums, field_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,expansion", [(65, 0), (65, 1), (77, 0)])
def test_fp64_ragged_rows_match_oracle(n, expansion):
    """Fields, local energies, lines, a field line and the spectrum in double."""
    import coolbubble_b200 as cb
    L, c = n / 4.0, 4.0
    dt = 0.1 * L / n
    phi0 = bubbles(3, n, L, c, 6, seed=7)
    kw = dict(expansion=expansion, mpl=10.0)
    o, ref = _oracle_run(3, n, L, c, dt, phi0, None, 20, 10, **kw)
    s = cb.Bubble(cb.make_params(3, n, L, c, dt, **kw), phi0)
    np.testing.assert_array_equal(s.phi, phi0.reshape(-1))
    for r in ref:
        check_sums(s.step(10, sums=True, local=True), r, n ** 3)
    line = s.line(5, 3, n - 1)
    f, fo = s.fields(), o.fields()
    for k in ("phi", "pi", "ekin", "egrad", "epot"):
        assert field_err(f[k], fo[k]) <= FIELD_TOL, k
    np.testing.assert_array_equal(line, np.roll(f["phi"].reshape(n, n, n)[:, 3, n - 1], -5))
    np.testing.assert_array_equal(s.fields_f32()["pi"], f["pi"].astype(np.float32))
    if n == 77:   # 7 * 11: the sizes the transform takes
        (pw, ws, _), (opw, ows, _) = s.spectrum_sums(), o.spectrum()
        np.testing.assert_array_equal(ws, ows)
        big = opw > 1e-8 * opw.max()
        np.testing.assert_allclose(pw[big], opw[big], rtol=1e-10)


@pytest.mark.parametrize("n,prec,expansion", [
    (65, "fp32c", 0), (66, "fp32c", 0), (67, "fp32c", 1), (129, "fp32c", 0), (130, "fp32c", 0), (131, "fp32c", 0),
    (65, "fp64", 0), (65, "fp64", 1), (129, "fp64", 0)])
def test_ragged_rows_equal_generic_kernel(n, prec, expansion, monkeypatch):
    """One, two and three sites in a row's last vector; one- and two-step passes
    and multi-step expanding launches; fields bit for bit (float expanding runs:
    to rounding of the Friedmann sums' order)."""
    import coolbubble_b200 as cb
    L = n / 8.0
    p = cb.make_params(3, n, L, 4.0, 0.1 * L / n, precision=prec, memorysave=1, expansion=expansion, mpl=10.0)
    phi0 = 0.4 + smooth_noise(3, n, 0.1, seed=3)
    pi0 = smooth_noise(3, n, 0.05, seed=4)
    monkeypatch.setenv("CB_TEMPORAL_BLOCK", "2")
    fast = cb.Bubble(p, phi0, pi0)
    monkeypatch.setenv("CB_STEP_PATH", "generic")
    generic = cb.Bubble(p, phi0, pi0)
    monkeypatch.undo()
    for k in (1, 4, 9):
        a, b = fast.step(k, sums=True), generic.step(k, sums=True)
    fa, fb = fast.fields(), generic.fields()
    for key in ("phi", "pi"):
        if expansion and prec == "fp32c":
            assert field_err(fa[key], fb[key]) <= 14 * 2.0 ** -23, key
        else:
            np.testing.assert_array_equal(fa[key], fb[key])
    for key in ("etot", "ekin", "egrad", "epot", "a", "etot_var", "avphi_var"):
        assert abs(a[key] - b[key]) <= (2.0 ** -21 if prec == "fp32c" else 1e-12) * abs(b[key]), key


@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
def test_ragged_start_built_on_the_device(prec):
    """A start drawn by cb_create_from_seed lands in the padded rows as the host's does."""
    import coolbubble_b200 as cb
    from coolbubble_b200.ic import initial_condition
    from coolbubble_b200.serving import create_from_seed, ic_params
    n, L = 66 if prec == "fp32c" else 65, 16.0
    p = cb.make_params(3, n, L, 4.0, 0.1 * L / n, precision=prec, memorysave=1)
    a = create_from_seed(p, ic_params(mode=1, n_bubbles=4))
    phi0, pi0, _ = initial_condition(p, mode=1, n_bubbles=4)
    b = cb.Bubble(p, phi0, pi0)
    for s in (a, b):
        s.step(6, sums=True)
    # the starts agree to a few units in the last place; pi gathers k dt times the
    # Laplacian's 12 / dx^2 of that
    tol = 1e-12 if prec == "fp64" else 6 * 2.0 ** -23
    most = tol * np.abs(b.phi).max()
    assert np.abs(a.phi - b.phi).max() <= most
    assert np.abs(a.pi - b.pi).max() <= 6 * (0.1 * L / n) * 12 / (L / n) ** 2 * most


@pytest.mark.parametrize("n,expansion", [(64, 0), (64, 1), (65, 0), (65, 1)])
def test_line_without_local_arrays_equals_line_with_them(n, expansion):
    """The reporting step's sums in double, with and without the local energy
    arrays (two variants of the staged kernel): each term within a few roundings,
    N of them added."""
    import coolbubble_b200 as cb
    L = n / 10.0   # dx^2 no power of two
    p = cb.make_params(3, n, L, 4.0, 0.1 * L / n, expansion=expansion, mpl=10.0)
    start = 0.4 + smooth_noise(3, n, 0.1, seed=5), smooth_noise(3, n, 0.05, seed=6)
    a, b = cb.Bubble(p, *start), cb.Bubble(p, *start)
    la, lb = a.step(3, sums=True, local=False), b.step(3, sums=True, local=True)
    tol = (n ** 3 + 16) * 2.0 ** -53
    for key in ("etot", "ekin", "egrad", "epot", "etot_var", "ekin_var", "egrad_var", "epot_var", "avphi_var",
                "avphip_var", "a", "ekin_half_prev"):
        assert abs(la[key] - lb[key]) <= tol * abs(lb[key]), key
    for key in ("avphi", "avphip"):
        assert abs(la[key] - lb[key]) <= tol * (n ** 3 * lb[key + "_var"]) ** 0.5, key
    np.testing.assert_array_equal(a.phi, b.phi)
