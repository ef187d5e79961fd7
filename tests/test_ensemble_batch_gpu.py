"""Ensembles stepped in batches: members of every form of row, sizes mixed in
one launch, against their solo runs, bit for bit in the fields."""
import numpy as np
import pytest

from ic_helpers import smooth_noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
def test_batched_members_equal_their_solo_runs(prec):
    import coolbubble_b200 as cb
    from coolbubble_b200.ensemble import Ensemble
    # whole rows of 8, 16, 32 lanes; vectors; site by site; dx^2 that divides in one, two operations and neither
    specs = [(32, 4.0), (64, 8.0), (128, 16.0), (64, 6.4), (200, 20.0), (256, 32.0), (101, 10.1), (502, 30.0), (5, 0.5)]
    made = []
    for i, (n, L) in enumerate(specs):
        p = cb.make_params(2, n, L, 2.0 + i % 3, 0.1 * L / n, precision=prec, memorysave=1)
        made.append((p, 0.3 + smooth_noise(2, n, 0.1, seed=i), smooth_noise(2, n, 0.05, seed=90 + i)))
    mix = [cb.Bubble(*m) for m in made]
    solo = [cb.Bubble(*m) for m in made]
    mix[2].step(3, sums=False)   # another buffer state than the others'
    solo[2].step(3, sums=False)
    ens = Ensemble(mix)
    for nsteps, every in ((7, 0), (85, 40), (1, 1), (40, 13)):
        lines = ens.step(nsteps, every)
        for i, s in enumerate(solo):
            ref, done = [], 0
            while every and done + every <= nsteps:
                ref.append(s.step(every, sums=True))
                done += every
            if done < nsteps:
                s.step(nsteps - done, sums=False)
            assert len(lines[i]) == len(ref)
            for got, want in zip(lines[i], ref):
                assert got["t"] == want["t"] and got["a"] == want["a"]
                for key in ("etot", "ekin", "egrad", "epot", "etot_var", "avphi_var"):
                    # the same terms, added in double in another order
                    assert abs(got[key] - want[key]) <= s.N * 2.0 ** -52 * abs(want[key]), (i, key)
    for i, (m, s) in enumerate(zip(mix, solo)):
        fa, fb = m.fields(), s.fields()
        np.testing.assert_array_equal(fa["phi"], fb["phi"], err_msg=str(specs[i]))
        np.testing.assert_array_equal(fa["pi"], fb["pi"], err_msg=str(specs[i]))
        assert m.sums()["t"] == s.sums()["t"] and m.counters()[1] == s.counters()[1]


@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
def test_large_members_step_as_their_solo_runs(prec):
    """A lattice that fills the GPU by itself takes its own launches, beside the
    batch of the small ones."""
    import coolbubble_b200 as cb
    from coolbubble_b200.ensemble import Ensemble
    made = []
    for n in (2048 if prec == "fp64" else 3072, 64, 64):
        p = cb.make_params(2, n, n / 8.0, 4.0, 0.0125, precision=prec, memorysave=1)
        rng = np.random.default_rng(n)
        made.append((p, 0.3 + 0.1 * rng.random(n * n), 0.05 * rng.standard_normal(n * n)))
    mix, solo = [cb.Bubble(*m) for m in made], [cb.Bubble(*m) for m in made]
    ens = Ensemble(mix)
    for nsteps, every in ((6, 1), (40, 40)):
        lines = ens.step(nsteps, every)
        for got, s in zip(lines, solo):
            want = [s.step(every, sums=True) for _ in range(nsteps // every)]
            for a, b in zip(got, want):
                assert a["t"] == b["t"] and abs(a["etot"] - b["etot"]) <= s.N * 2.0 ** -52 * abs(b["etot"])
    assert mix[0].counters() == solo[0].counters()
    for m, s in zip(mix, solo):
        fa, fb = m.fields(), s.fields()
        for key in ("phi", "pi"):
            np.testing.assert_array_equal(fa[key], fb[key])


def test_plan_tells_which_members_are_batched():
    """Threads of a block for every member of a batch, one number per batch, whatever
    its size class; none for members on their own streams."""
    import coolbubble_b200 as cb
    from coolbubble_b200.ensemble import Ensemble

    def run(d, n, prec):
        p = cb.make_params(d, n, n / 8.0, 4.0, 0.0125, precision=prec, memorysave=1)
        return cb.Bubble(p, np.zeros(n ** d))

    runs = [run(2, 1000, "fp32c"), run(2, 64, "fp32c"), run(2, 400, "fp32c"), run(2, 250, "fp64"), run(2, 2048, "fp64"),
            run(3, 16, "fp64"), run(1, 64, "fp64")]
    plans = [Ensemble(runs).plan(i) for i in range(len(runs))]
    assert all(threads in (128, 256, 512) for _, threads in plans[:4])
    assert plans[0][0] == 0                     # beyond the classes, and batched all the same
    assert plans[0][1] == plans[2][1]           # one batch: rows of vectors, float
    assert plans[4:] == [(0, 0)] * 3


def test_batched_members_that_divide_by_division_equal_their_solo_runs():
    """dx^2 without a two-operation division: a batch of its own."""
    import coolbubble_b200 as cb
    from coolbubble_b200.ensemble import Ensemble
    made = []
    for i, n in enumerate((64, 200, 101, 500)):
        p = cb.make_params(2, n, n * 0.17, 4.0, 0.017, precision="fp64", memorysave=1)
        made.append((p, 0.3 + smooth_noise(2, n, 0.1, seed=i), smooth_noise(2, n, 0.05, seed=50 + i)))
    mix, solo = [cb.Bubble(*m) for m in made], [cb.Bubble(*m) for m in made]
    Ensemble(mix).step(23, 0)
    for m, s in zip(mix, solo):
        s.step(23, sums=False)
        a, b = m.fields(), s.fields()
        for key in ("phi", "pi"):
            np.testing.assert_array_equal(a[key], b[key])
