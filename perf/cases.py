"""Timed cases: what a program that uses this library has it do.

Three kinds of work, each through the package's public entry points:

  run       one lattice (Bubble): the stretch of a run between two snapshots. The energy line is read every
            `every` steps (the reference's main loop writes one every 40), and at the end the program takes the
            power spectrum, where it writes one, and the float snapshot of phi and pi, into page-locked buffers
            that it keeps (cb_get_fields_f32, the data that OutField stores).
  ensemble  independent two-dimensional lattices stepped together (Ensemble), their lines and their snapshots.
  serve     requests through the serving pool: submitted together, each started from its seed, stepped to its
            end, its lines and fields collected.

Precision, dimension, background (static or expanding), lattice size and lattice spacing vary: n that are powers
of two, n that are not and odd n; a spacing dx whose square is a power of two, and one whose square is not.
"""
import math

import numpy as np
import torch

import coolbubble_b200 as cb
from coolbubble_b200 import _lib as L
from coolbubble_b200.ensemble import Ensemble
from coolbubble_b200.serving import DONE, Pool, ic_params

#: The columns of an energy line, as the program appends it to its table.
COLUMNS = ("t", "a", "H", "C", "etot", "ekin", "egrad", "epot", "etot_var", "ekin_var", "egrad_var", "epot_var",
           "avphi", "avphi_var", "avphip", "avphip_var")


def _run(name, d, n, dx, c, precision, steps, start, expansion=0, every=40, spectrum=False):
    return {"name": name, "kind": "run", "d": d, "n": n, "dx": dx, "c": c, "precision": precision, "steps": steps,
            "every": every, "start": start, "expansion": expansion, "spectrum": spectrum}


def listed():
    return [
        # the smallest call: a caller that drives a one-dimensional lattice one step at a time and reads it each time
        _run("one step, d1 n1024 fp64", 1, 1024, 0.1, 4.0, "fp64", 1, "bubbles", every=1),
        # the reference's example run: 512^2, five bubbles, FP64 throughout, with spectra
        _run("d2 n512 fp64 bubbles", 2, 512, 0.0625, 4.0, "fp64", 200, "bubbles", spectrum=True),
        # an ordinary two-dimensional lattice of a size that is no power of two
        _run("d2 n1000 fp32c thermal", 2, 1000, 0.1, 2.0, "fp32c", 400, "thermal"),
        # a large two-dimensional lattice in double, with a spacing that makes the force divide
        _run("d2 n3072 fp64 thermal", 2, 3072, 0.1, 2.0, "fp64", 120, "thermal"),
        # a small three-dimensional lattice of the kind that the serving stream carries
        _run("d3 n192 fp32c static", 3, 192, 0.125, 4.0, "fp32c", 400, "bubbles", spectrum=True),
        # a ragged size: rows that are no whole number of 16-byte vectors
        _run("d3 n250 fp32c static", 3, 250, 0.128, 2.0, "fp32c", 200, "thermal"),
        # the plain double path on a static background
        _run("d3 n256 fp64 static", 3, 256, 0.125, 2.0, "fp64", 200, "thermal"),
        # the expanding run: 256^3, eight bubbles, the background updated every step; both precisions
        _run("d3 n256 fp32c expanding", 3, 256, 0.125, 4.0, "fp32c", 200, "bubbles", expansion=1, spectrum=True),
        _run("d3 n256 fp64 expanding", 3, 256, 0.125, 4.0, "fp64", 200, "bubbles", expansion=1, spectrum=True),
        # the largest: the 512^3 thermal run
        _run("d3 n512 fp32c thermal", 3, 512, 0.125, 2.0, "fp32c", 400, "thermal", spectrum=True),
        # an ensemble of two-dimensional lattices of three sizes (a parameter scan)
        {"name": "ensemble of 48, fp32c", "kind": "ensemble", "members": 48, "precision": "fp32c", "steps": 400,
         "every": 40},
        # a burst of requests to the serving pool
        {"name": "serve 8 requests", "kind": "serve", "requests": 8, "n_most": 192, "steps": 400, "every": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """Whether the spectrum takes this size (prime factors up to 13)."""
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    kind = rng.choice(["run"] * 8 + ["ensemble", "serve"])
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(6, 48), "precision": rng.choice(["fp32c", "fp32c", "fp64"]),
                "steps": 40 * rng.randint(2, 10), "every": 40}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(3, 10), "n_most": rng.choice([96, 128, 160, 192]),
                "steps": 40 * rng.randint(2, 10), "every": 40}
    d = rng.choice([1, 2, 2, 3, 3, 3])
    lo, hi = {1: (256, 1 << 20), 2: (48, 4096), 3: (40, 400)}[d]
    n = _log_int(rng, lo, hi)
    grain = rng.choice([1, 2, 4, 16, 64])   # odd sizes, even ones, whole vectors, whole tiles
    n = max(grain, n // grain * grain)
    c = _run("", d, n, rng.choice([0.0625, 0.1, 0.125]), rng.choice([2.0, 4.0, 6.0]), rng.choice(["fp64", "fp32c"]),
             40 * _log_int(rng, 1, 10), rng.choice(["bubbles", "thermal"]),
             expansion=1 if d == 3 and rng.random() < 0.5 else 0, spectrum=_smooth(n) and n <= 4096 and rng.random() < 0.5)
    if c["expansion"]:
        c["start"] = "bubbles"
    del c["name"]
    return c


# ---- inputs --------------------------------------------------------------------------------------------------------

def _fields(seed, d, n, dx, c, start):
    """phi and pi at t = 0, of float values held as doubles (so both precisions take the same start): bubbles of
    true vacuum at random places, or a thermal state (Gaussian modes of variance T / omega^2 and T)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    box = n * dx
    shape = (n,) * d
    if start == "bubbles":
        # profile, radius and wall width as the reference fits them for a given c
        phic, r, w = 0.997 * (1 - math.exp(-c * 0.688)), 0.823 * c ** 0.203 * (1.3 if d == 3 else 1.0), 0.496 * c ** -0.531
        at = torch.rand(8 if d == 3 else 5, d, generator=gen, device="cuda", dtype=torch.float64) * box
        x = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * dx
        phi = torch.zeros(shape, device="cuda", dtype=torch.float64)
        for b in at:
            r2 = torch.zeros((1,) * d, device="cuda", dtype=torch.float64)
            for ax in range(d):
                s = (x - b[ax]).abs()
                s = torch.minimum(s, box - s)
                r2 = r2 + (s * s).reshape((1,) * ax + (n,) + (1,) * (d - 1 - ax))
            phi = torch.maximum(phi, phic / 2 * (torch.tanh((r - r2.sqrt()) / w) + 1))
        pi = torch.zeros_like(phi)
    else:
        temp = 0.05 * math.sqrt(2 * (c + 6))
        k = 2 * math.pi * torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
        one = 4 / dx ** 2 * torch.sin(k / 2) ** 2
        om2 = torch.full((1,) * d, 2 * c, device="cuda", dtype=torch.float64)
        for ax in range(d):
            last = ax == d - 1
            om2 = om2 + one[: n // 2 + 1 if last else n].reshape((1,) * ax + (-1,) + (1,) * (d - 1 - ax))
        noise = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64) * math.sqrt(temp / dx ** d)
        phi = torch.fft.irfftn(torch.fft.rfftn(noise) / om2.sqrt(), s=shape)
        pi = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64) * math.sqrt(temp / dx ** d)
    return phi.float().double(), pi.float().double()


def _members(case, seed):
    """The ensemble's lattices: sizes in equal thirds, c over its range, bubbles and thermal starts in turn."""
    rng = np.random.default_rng(seed)
    out = []
    for m in range(case["members"]):
        out.append({"d": 2, "n": (128, 256, 512)[m % 3], "dx": 0.125, "c": float(rng.uniform(1, 8)), "expansion": 0,
                    "precision": case["precision"], "steps": case["steps"], "every": case["every"],
                    "start": "bubbles" if m % 2 else "thermal", "seed": int(rng.integers(1 << 40))})
    return out


def _requests(case, seed):
    """The burst: d in {2, 3}, several sizes, half of the three-dimensional runs expanding, each with its own seeds."""
    rng = np.random.default_rng(seed)
    out = []
    for m in range(case["requests"]):
        d = 3 if m % 2 else 2
        n = (case["n_most"], 64, case["n_most"] // 2 + 1, 96)[(m // 2) % 4]
        p = _params({"d": d, "n": n, "dx": 0.125, "c": (2.0, 4.0, 6.0)[m % 3], "precision": "fp32c",
                     "expansion": int(d == 3 and m % 4 == 1)})
        ic = ic_params(mode=-3 if m % 4 == 3 and _smooth(n) else 1, n_bubbles=5, trad=0.05,
                       position_seed=int(rng.integers(1, 2 ** 31)), thermal_seed=int(rng.integers(1, 2 ** 62)))
        out.append((p, ic, case["steps"] * (1 + m % 2), n ** d))
    return out


def _params(m):
    return cb.make_params(m["d"], m["n"], m["n"] * m["dx"], m["c"], 0.1 * m["dx"], expansion=m["expansion"], mpl=10.0,
                          precision=m["precision"], memorysave=1)


def _host(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _bubble(m, seed):
    phi, pi = _fields(seed, m["d"], m["n"], m["dx"], m["c"], m["start"])
    up = _host(2 * phi.numel(), torch.float64)
    torch.from_numpy(up[: phi.numel()]).copy_(phi.reshape(-1))
    torch.from_numpy(up[phi.numel():]).copy_(pi.reshape(-1))
    return cb.Bubble(_params(m), up[: phi.numel()], up[phi.numel():])


def prepare(case, seed):
    if case["kind"] == "serve":
        return {"case": case, "requests": _requests(case, seed), "pool": Pool(150 * 10 ** 9, 64)}
    if case["kind"] == "ensemble":
        ms = _members(case, seed)
        runs = [_bubble(m, m["seed"]) for m in ms]
        sites = sum(r.N for r in runs)
        return {"case": case, "runs": runs, "ensemble": Ensemble(runs), "phi": _host(sites, torch.float32),
                "pi": _host(sites, torch.float32)}
    s = _bubble(case, seed)
    return {"case": case, "bubble": s, "phi": _host(s.N, torch.float32), "pi": _host(s.N, torch.float32)}


# ---- one pass ------------------------------------------------------------------------------------------------------

def _snapshot(s, phi, pi):
    L.check(L.lib.cb_get_fields_f32(s._h, L.fptr(phi), L.fptr(pi), None, None, None), s._h)


def _table(lines):
    return np.array([[line[c] for c in COLUMNS] for line in lines])


def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        pool = state["pool"]
        ids = [pool.submit(p, ic, nt, sums_every=case["every"], want_fields=True) for p, ic, nt, _ in state["requests"]]
        out = []
        for rid, (_, _, nt, sites) in zip(ids, state["requests"]):
            pool.wait(rid)
            r = pool.result(rid, n_sites=sites, max_lines=nt // case["every"])
            if r["state"] != DONE:
                raise RuntimeError("request failed: " + r["err"])
            out.append({"lines": _table(r["lines"]), "phi": r["phi"], "pi": r["pi"]})
        return out
    if case["kind"] == "ensemble":
        lines = state["ensemble"].step(case["steps"], case["every"])
        at = 0
        for s in state["runs"]:
            _snapshot(s, state["phi"][at: at + s.N], state["pi"][at: at + s.N])
            at += s.N
        return {"lines": np.concatenate([_table(x) for x in lines]), "phi": state["phi"], "pi": state["pi"]}
    s = state["bubble"]
    lines = [s.step(case["every"]) for _ in range(case["steps"] // case["every"])]
    out = {"lines": _table(lines)}
    if case["spectrum"]:
        rows = s.ComputePowerSpectrum()
        out["k"], out["power"] = rows[:, 0], rows[:, 2]
    _snapshot(s, state["phi"], state["pi"])
    return dict(out, phi=state["phi"], pi=state["pi"])


def work(case):
    """Each field read once and written once in its own precision, and the float snapshot written; per site and step
    the Laplacian (3 d), V' (7), force, kick and drift (7)."""
    if case["kind"] == "run":
        parts = [(case["n"] ** case["d"], case["d"], case["steps"], 8 if case["precision"] == "fp64" else 4)]
    elif case["kind"] == "ensemble":
        parts = [(m["n"] ** 2, 2, m["steps"], 8 if m["precision"] == "fp64" else 4) for m in _members(case, 1)]
    else:
        parts = [(sites, p.d, nt, 4) for p, _, nt, sites in _requests(case, 1)]
    return {"bytes": sum(N * (4 * size + 8) for N, _, _, size in parts),
            "flops": sum(N * steps * (3 * d + 14) for N, d, steps, _ in parts)}


# ---- the same in 64 bits, in torch ---------------------------------------------------------------------------------

def _evolve(m, seed):
    """The leapfrog run of one lattice: its lines and its fields after m["steps"] steps."""
    d, n, dx, c = m["d"], m["n"], m["dx"], m["c"]
    phi, pi = _fields(seed, d, n, dx, c, m["start"])
    dt, cell = 0.1 * dx, (dx / (n * dx)) ** d
    mpl2, grows = 3.0 * 10.0 * 10.0, bool(m["expansion"])

    def pot(f):
        return c * f ** 2 - (2 * c + 4) * f ** 3 + (c + 3) * f ** 4 + 1.0

    def force(f, a):
        out = sum(f.roll(-1, ax) + f.roll(1, ax) for ax in range(d)).sub_(f, alpha=2 * d).mul_(a ** (d - 2) / dx ** 2)
        return out.sub_(f * (2 * c + f * (-3 * (2 * c + 4) + f * (4 * (c + 3)))), alpha=a ** d)

    def grad(f, h):
        return sum(((f.roll(-1, ax) - f) / h).square_() for ax in range(d)).mul_(0.5)

    def ddot(a, ek, ep):
        return -a * (2 * ek - ep) / mpl2 if grows else 0.0

    ek, ep, eg = (float(x.sum()) * cell for x in (0.5 * pi * pi, pot(phi), grad(phi, dx)))
    a, H, t = 1.0, math.sqrt((ek + ep + eg) / mpl2) if grows else 0.0, 0.0
    ap = a * H - 0.5 * dt * ddot(a, ek, ep)
    pi = pi - 0.5 * dt * force(phi, a)
    half = float((pi * pi).sum()) * 0.5 * (a - 0.5 * dt * ap) ** (-2 * d) * cell
    lines = []
    for it in range(1, m["steps"] + 1):
        wanted = it % m["every"] == 0
        a_kin = a + 0.5 * dt * ap
        if wanted and not grows:
            half = float((pi * pi).sum()) * 0.5 * a_kin ** (-2 * d) * cell
        pi.add_(force(phi, a), alpha=dt)
        if grows or wanted:
            now = float((pi * pi).sum()) * 0.5 * a_kin ** (-2 * d) * cell
            ek, half, was = 0.5 * (half + now), now, a
            v = pot(phi)
            ep = float(v.sum()) * cell
            prev, ap = ap, ap + dt * ddot(a, ek, ep)
            a = a + dt * ap
            H = 0.5 * (prev + ap) / was
        t += dt
        if wanted:
            g, e, vel = grad(phi, was * dx), 0.5 * a_kin ** (-2 * d) * pi * pi, pi * a_kin ** -d
            eg = float(g.sum()) * cell
            tot = ek + ep + eg
            sq = [float(x.square().sum()) * cell ** 2 for x in (e + g + v, e, g, v, phi, vel)]
            lines.append([t, a, H, H * H - tot / mpl2 if grows else 0.0, tot, ek, eg, ep, sq[0], sq[1], sq[2], sq[3],
                          float(phi.sum()) * cell, sq[4], float(vel.sum()) * cell, sq[5]])
            del g, e, vel
        phi.add_(pi, alpha=dt * (0.5 * (was + a)) ** -d if grows else dt)
    return np.array(lines), phi, pi


def _spectrum(m, phi):
    """(k, power) of the shells that hold modes: |k| in units of 2 pi / box cut to its whole part."""
    d, n, dx = m["d"], m["n"], m["dx"]
    box = n * dx
    half = torch.fft.rfftn(phi).abs().square_()
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    i = torch.where(i <= n // 2, i, i - n)
    r2 = torch.zeros((1,) * d, device="cuda", dtype=torch.float64)
    for ax in range(d):
        x = i[: n // 2 + 1] if ax == d - 1 else i
        r2 = r2 + (x * x).reshape((1,) * ax + (-1,) + (1,) * (d - 1 - ax))
    r = r2.sqrt().expand(half.shape)
    w = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    w[0] = 1.0
    w[n // 2] = 1.0
    w = w.expand(half.shape)
    bins = r.long().reshape(-1)
    dk = 2 * math.pi / box
    pref = {1: 1 / math.pi, 2: 1 / (2 * math.pi), 3: 1 / (2 * math.pi ** 2)}[d] * dx ** (2 * d) / box ** d

    def add(x):
        return torch.zeros(int(bins.max()) + 1, device="cuda", dtype=torch.float64).index_add_(0, bins, x.reshape(-1))

    weight = add(w)
    on = weight > 0
    return ((add(w * r * dk) / weight)[on].cpu().numpy(),
            (add(w * (r * dk) ** d * half * pref) / weight)[on].cpu().numpy())


def exact(case, seed):
    if case["kind"] == "serve":
        return None   # the starts are drawn by the library from its seeds
    if case["kind"] == "ensemble":
        all_ = [_evolve(m, m["seed"]) for m in _members(case, seed)]
        return {"lines": np.concatenate([x[0] for x in all_]), "phi": torch.cat([x[1].reshape(-1) for x in all_]),
                "pi": torch.cat([x[2].reshape(-1) for x in all_])}
    lines, phi, pi = _evolve(case, seed)
    out = {"lines": lines}
    if case["spectrum"]:
        out["k"], out["power"] = _spectrum(case, phi)
    return dict(out, phi=phi.reshape(-1), pi=pi.reshape(-1))
