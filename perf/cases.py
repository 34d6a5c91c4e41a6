"""The work that programs give this library, as timed cases.

Three kinds of call, over the sizes of the repository's own workloads (216 to
96,000 waters: 648 to 288,000 atoms) and both precision forms:

* "solve": one single-point polarization solve on host buffers
  (Context.solve_host with pinned arrays, the list built anew because the
  positions are unrelated to those before): coordinates in, both sets of
  induced dipoles and the polarization energy out.
* "batch": many small boxes of uneven size solved together by a batch plan
  (lib.Batch), and every box's dipoles read back.
* "step": two consecutive steps of dynamics with every non-bonded term (new
  coordinates 0.01 A from the last ones, a solve started from the previous
  dipoles, the gradient of the polarization energy, the permanent-multipole
  and the van der Waals energy and gradient), with or without the virials.
* "md": velocity-Verlet dynamics on the device (Context.md_verlet) from given
  coordinates and velocities.

exact() states the same results in plain torch FP64: brute-force pairs, the
smooth-PME sums with torch's FFT, conjugate gradients to 1e-13, and gradients
by differentiating the (variational) energies.
"""
import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

# many independent systems run as parallel graph branches; the default of 8
# hardware queues would serialise them (read when the CUDA context is made)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

POLEPS = 1e-6          # the CG stop of the benchmark, the tests and the server
MOVE = 0.01            # A RMS per coordinate between the steps of a "step" case
DT = 0.001             # ps
EXACT_ATOMS = 100_000  # exact() of a case with gradients


def _package():
    name = "tinker_hp_b200"
    if name not in sys.modules:
        d = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tinker-hp_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        sys.modules[name] = m = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(m)
    import tinker_hp_b200.lib
    import tinker_hp_b200.water
    return sys.modules[name]


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # one small molecule-sized box at a time: latency and launches
        {"name": "solve_648_fp64", "kind": "solve", "nw": 216, "mixed": False},
        {"name": "solve_1944_mixed", "kind": "solve", "nw": 648, "mixed": True},
        # a box whose atom count is no multiple of anything
        {"name": "solve_9003_mixed", "kind": "solve", "nw": 3001, "mixed": True},
        # the dynamics box of the repository's first configuration, as single points
        {"name": "solve_32k_mixed", "kind": "solve", "nw": 10800, "mixed": True},
        {"name": "solve_32k_fp64", "kind": "solve", "nw": 10800, "mixed": False},
        # the benchmark's box, in both forms
        {"name": "solve_288k_mixed", "kind": "solve", "nw": 96000, "mixed": True},
        {"name": "solve_288k_fp64", "kind": "solve", "nw": 96000, "mixed": False},
        # uneven small boxes together (screening many small systems)
        {"name": "batch_32_mixed", "kind": "batch", "count": 32, "nmin": 300, "nmax": 6000, "mixed": True},
        {"name": "batch_12_fp64", "kind": "batch", "count": 12, "nmin": 300, "nmax": 6000, "mixed": False},
        # dynamics driven from outside: all non-bonded terms per step
        {"name": "step_96k_mixed", "kind": "step", "nw": 32000, "mixed": True, "virial": False},
        {"name": "step_4113_fp64_virial", "kind": "step", "nw": 1371, "mixed": False, "virial": True},
        # dynamics on the device
        {"name": "md_32k_fp64", "kind": "md", "nw": 10800, "mixed": False, "steps": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "step", "md"])
    mixed = rng.random() < 0.5
    if kind == "solve":
        return {"kind": "solve", "nw": _log_int(rng, 216, 96000), "mixed": mixed}
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 4, 32), "nmin": 300, "nmax": _log_int(rng, 1500, 6000),
                "mixed": mixed}
    if kind == "step":
        return {"kind": "step", "nw": _log_int(rng, 300, 32000), "mixed": mixed, "virial": rng.random() < 0.3}
    return {"kind": "md", "nw": _log_int(rng, 300, 10800), "mixed": mixed, "steps": rng.randint(2, 4)}


# ---- inputs and the timed calls ------------------------------------------------

def _box(nw, seed):
    return _package().water.make_water_box(nw, seed_lattice=2 * seed + 1, seed_orient=2 * seed + 2)


def _batch_boxes(case, seed):
    """Uneven boxes as the batch workload makes them (log-uniform atom counts,
    small edges widened to the list cutoff); the sizes come from the case, the
    coordinates from the seed."""
    water = _package().water
    sizes = water.batch_sizes(case["count"], case["nmin"], case["nmax"], seed=4003)
    return [water.make_water_box(nw, edge=max(water.box_edge(nw), water.min_box_edge()),
                                 seed_lattice=1000 * seed + 2 * q, seed_orient=1000 * seed + 2 * q + 1)
            for q, nw in enumerate(sizes)]


def _frames(ws, seed):
    """The two coordinate sets of a "step" case after the box's own."""
    rng = np.random.default_rng([seed, 7])
    p1 = ws.positions() + rng.normal(0.0, MOVE, (ws.n, 3))
    return [p1, p1 + rng.normal(0.0, MOVE, (ws.n, 3))]


def _pinned(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64).pin_memory().numpy()


def _columns(p):
    return [_pinned(p[:, d]) for d in range(3)]


def _context(ws, case):
    lib = _package().lib
    return lib.Context(ws, precision=lib.MIXED if case["mixed"] else lib.FP64, poleps=POLEPS)


def _step(s, q):
    ctx, b = s["ctx"], s["buf"][q]
    ctx.set_positions(*s["frames"][q])
    epol = ctx.solve(s["previous"])["epol"]
    _, g = ctx.gradient(out=b[0])
    em, gm = ctx.empole1(out=b[1])
    ev, gv = ctx.ehal1(out=b[2])
    out = {"energies": np.array([epol, em, ev]), "dep": g, "dem": gm, "dev": gv}
    if s["virial"]:
        out["vir"] = np.stack([ctx.virial(), ctx.empole_virial(), ctx.ehal_virial()])
    return out


def prepare(case, seed):
    pkg = _package()
    lib = pkg.lib
    if case["kind"] == "solve":
        ws = _box(case["nw"], seed)
        return {"kind": "solve", "ctx": _context(ws, case), "xyz": _columns(ws.positions()),
                "out": (_pinned(np.zeros((ws.n, 3))), _pinned(np.zeros((ws.n, 3))))}
    if case["kind"] == "batch":
        ctxs = [_context(ws, case) for ws in _batch_boxes(case, seed)]
        plan = lib.Batch(ctxs)
        tuning = 0
        while plan.tuning() is None and tuning < 16:  # the plan settles its launch shape at start-up
            plan.solve()
            tuning += 1
        return {"kind": "batch", "ctxs": ctxs, "plan": plan}
    ws = _box(case["nw"], seed)
    ctx = _context(ws, case)
    if case["kind"] == "md":
        mass = pkg.water.masses(ws)
        vel = pkg.water.maxwell_velocities(mass, 300.0, seed=seed)
        return {"kind": "md", "ctx": ctx, "xyz": _columns(ws.positions()), "mass": mass, "vel": vel,
                "steps": case["steps"]}
    ctx.set_virial(case["virial"])
    s = {"kind": "step", "ctx": ctx, "virial": case["virial"], "previous": lib.GUESS_PREVIOUS,
         "frames": [_columns(p) for p in _frames(ws, seed)] + [_columns(ws.positions())],
         "buf": [[_pinned(np.zeros((ws.n, 3))) for _ in range(3)] for _ in range(3)]}
    _step(s, 2)  # the dynamics is under way: lists and dipoles of the step before
    return s


def run(s):
    if s["kind"] == "solve":
        s["ctx"].invalidate_list()
        uind, uinp, info = s["ctx"].solve_host(*s["xyz"], out=s["out"])
        return {"uind": uind, "uinp": uinp, "epol": info["epol"]}
    if s["kind"] == "batch":
        infos = s["plan"].solve()
        dip = [c.dipoles() for c in s["ctxs"]]
        return {"uind": np.concatenate([d[0] for d in dip]), "uinp": np.concatenate([d[1] for d in dip]),
                "epol": np.array([f["epol"] for f in infos])}
    if s["kind"] == "md":
        ctx = s["ctx"]
        ctx.invalidate_list()
        ctx.set_positions(*s["xyz"])
        vel, en, _ = ctx.md_verlet(s["steps"], DT, s["mass"], s["vel"])
        return {"pos": ctx.positions(), "vel": vel, "energies": en}
    return [_step(s, q) for q in range(2)]


# ---- work and tolerances -------------------------------------------------------

def _solve_flops(n, k3, iterations):
    """Floating-point operations of one solve from the path's per-unit counts:
    71.8 N interacting half-pairs (120 per matvec, 220 in the direct field),
    712 list candidates per atom (30 each), 3,500 per atom and 10 K^3 log2 K^3
    + 6 K^3 per reciprocal pass, 60 per atom in the CG vectors."""
    pairs = 71.8 * n
    recip = 3500.0 * n + 10.0 * k3 * math.log2(k3) + 6.0 * k3
    return (iterations + 1) * (120.0 * pairs + recip + 60.0 * n) + 220.0 * pairs + recip + 30.0 * 712.0 * n


def work(case):
    water, params = _package().water, _package().params
    if case["kind"] == "batch":
        sizes = water.batch_sizes(case["count"], case["nmin"], case["nmax"], seed=4003)
    else:
        sizes = [case["nw"]]
    flops = nbytes = 0.0
    for nw in sizes:
        n = 3 * nw
        edge = water.box_edge(nw)
        if case["kind"] == "batch":
            edge = max(edge, water.min_box_edge())
        k3 = float(params.pme_grid_size(edge)) ** 3
        # gradients: 71.8 N polarization and multipole pairs (about 800 and 500
        # operations), 152.6 N van der Waals pairs (60) and one reciprocal pass each
        forces = (71.8 * 1300.0 + 152.6 * 60.0 + 7000.0) * n + 20.0 * k3 * math.log2(k3)
        inputs = n * (3 + 13 + 3) * 8.0  # coordinates, multipoles, polarizability, Thole and damping
        if case["kind"] in ("solve", "batch"):
            flops += _solve_flops(n, k3, 9)
            nbytes += inputs + 48.0 * n
        elif case["kind"] == "step":
            flops += 2 * (_solve_flops(n, k3, 6) + forces)
            nbytes += 2 * (inputs + 72.0 * n)
        else:
            flops += (case["steps"] + 1) * (_solve_flops(n, k3, 8) + 71.8 * 800.0 * n)
            nbytes += (case["steps"] + 1) * (inputs + 48.0 * n)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # The mixed form's FP32 pair and grid sums differ between orders of summation
    # by 1.5e-7 to 3e-7 of the dipoles and gradients (the same inputs twice), a
    # few times that where the pair terms are rounded elsewhere.  The CG stops at
    # POLEPS in both forms, which leaves the dipoles 1.4e-5 to 2.1e-5 of their size
    # from exact(), the same for every implementation that takes the same number
    # of iterations.
    return {"rel": 1e-5, "max": 2e-4}


# ---- the same results in plain torch FP64 -------------------------------------

ELECTRIC = 332.063714
SQRT_PI = math.sqrt(math.pi)
CHUNK = 1 << 21  # pairs evaluated at a time


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), dtype=dtype, device="cuda")


class _System:
    """Fixed data of a water box on the GPU."""

    def __init__(self, ws):
        self.n, self.box = ws.n, _t(ws.box)
        self.a, self.cut, self.nfft = ws.aewald, ws.ewaldcut, ws.nfft
        self.pole = _t(ws.pole)
        self.iz, self.ix = _t(ws.zaxis, torch.int64), _t(ws.xaxis, torch.int64)
        self.bisector = _t(ws.axt == 2, torch.bool)[:, None]
        self.alpha, self.thole, self.pdamp = _t(ws.polarity), _t(ws.thole), _t(ws.pdamp)
        self.vdw = ws.vdw
        self.term = 4.0 / 3.0 * self.a ** 3 / SQRT_PI
        self.qfac = self._influence()

    def _influence(self):
        """exp(-pi^2 h^2/a^2) / (pi V h^2 B1 B2 B3) with the moduli of the
        order-5 splines and their aliasing correction (Essmann et al. 1995)."""
        mods, freq = [], []
        for d in range(3):
            nf = self.nfft[d]
            k = torch.arange(nf, device="cuda", dtype=torch.float64)
            w = torch.stack(_splines(torch.zeros(1, device="cuda", dtype=torch.float64), 5)).flatten()
            j = torch.arange(5, device="cuda", dtype=torch.float64)
            ph = 2.0 * math.pi / nf * k[:, None] * (j + 1.0)
            b = (w * torch.cos(ph)).sum(1) ** 2 + (w * torch.sin(ph)).sum(1) ** 2
            b = torch.where(b < 1e-7, 0.5 * (torch.roll(b, 1) + torch.roll(b, -1)), b)
            m = torch.where(k > nf // 2, k - nf, k)
            fac = math.pi * m / nf
            s1, s2 = torch.ones_like(m), torch.ones_like(m)
            for q in range(1, 51):
                for t in (fac / (fac + math.pi * q), fac / (fac - math.pi * q)):
                    s1, s2 = s1 + t ** 5, s2 + t ** 10
            mods.append(b * (s2 / s1) ** 2)
            freq.append(torch.where(k < (nf + 1) // 2, k, k - nf) / self.box[d])
        h2 = freq[2][:, None, None] ** 2 + freq[1][None, :, None] ** 2 + freq[0][None, None, :] ** 2
        e = -(math.pi / self.a) ** 2 * h2
        q = torch.exp(e) / (math.pi * self.box.prod() * h2 * mods[2][:, None, None] * mods[1][None, :, None]
                            * mods[0][None, None, :])
        q[0, 0, 0] = 0.0
        return torch.where(e > -50.0, q, torch.zeros_like(q))


def _splines(w, order):
    """The `order` nonzero cardinal B-splines at fraction w."""
    t = [1.0 - w, w]
    for k in range(3, order + 1):
        low = [torch.zeros_like(w)] + t + [torch.zeros_like(w)]
        # value i of order k from values i-1 and i of order k-1
        t = [((w + (k - 1 - i)) * low[i] + ((1 + i) - w) * low[i + 1]) / (k - 1) for i in range(k)]
    return t


def _spline_table(w, levels):
    """[n, levels, 5]: the order-5 splines and their derivatives."""
    rows = []
    for lev in range(levels):
        t = _splines(w, 5 - lev)
        for _ in range(lev):
            low = [torch.zeros_like(w)] + t + [torch.zeros_like(w)]
            t = [low[i] - low[i + 1] for i in range(len(t) + 1)]
        rows.append(torch.stack(t, -1))
    return torch.stack(rows, 1)


def _stencil(s, x, levels=3):
    """Grid indices [n, 125] and the three axes' spline tables."""
    idx, tab = [], []
    for d in range(3):
        f = x[:, d] / s.box[d]
        fr = s.nfft[d] * (f - torch.round(f.detach()) + 0.5)
        i0 = torch.clamp((fr.detach() - 1e-8).long(), 0, s.nfft[d] - 1)
        tab.append(_spline_table(fr - i0, levels))
        idx.append(torch.remainder(i0[:, None] - 4 + torch.arange(5, device="cuda"), s.nfft[d]))
    flat = (idx[2][:, :, None, None] * s.nfft[1] + idx[1][:, None, :, None]) * s.nfft[0] + idx[0][:, None, None, :]
    return flat.reshape(len(x), 125), tab


def _outer(tab, lx, ly, lz):
    return (tab[2][:, lz, :, None, None] * tab[1][:, ly, None, :, None] * tab[0][:, lx, None, None, :]).flatten(1)


def _spread(s, st, values):
    return torch.zeros(s.nfft[0] * s.nfft[1] * s.nfft[2], dtype=torch.float64, device="cuda").index_add(
        0, st[0].flatten(), values.flatten())


def _convolve(s, grid):
    shape = (s.nfft[2], s.nfft[1], s.nfft[0])
    return (torch.fft.ifftn(torch.fft.fftn(grid.view(shape)) * s.qfac, norm="forward").real).flatten()


def _spread_dipoles(s, st, mu):
    a = [s.nfft[d] / s.box[d] for d in range(3)]
    return _spread(s, st, a[0] * mu[:, :1] * _outer(st[1], 1, 0, 0) + a[1] * mu[:, 1:2] * _outer(st[1], 0, 1, 0)
                   + a[2] * mu[:, 2:] * _outer(st[1], 0, 0, 1))


def _gather_gradient(s, st, conv):
    c = conv[st[0]]
    return torch.stack([s.nfft[d] / s.box[d] * (c * _outer(st[1], *(1 if q == d else 0 for q in range(3)))).sum(1)
                        for d in range(3)], 1)


def _spread_poles(s, st, rp):
    a = [s.nfft[d] / s.box[d] for d in range(3)]
    v = rp[0][:, None] * _outer(st[1], 0, 0, 0)
    for d in range(3):
        v = v + a[d] * rp[1][:, d:d + 1] * _outer(st[1], *(int(q == d) for q in range(3)))
        for e in range(3):
            lev = [int(q == d) + int(q == e) for q in range(3)]
            v = v + a[d] * a[e] * rp[2][:, d, e, None] * _outer(st[1], *lev)
    return _spread(s, st, v)


def _rotate(s, x):
    """Charges, dipoles and quadrupoles in the box frame."""
    unit = lambda v: v / v.norm(dim=1, keepdim=True)
    u, v = x[s.iz] - x, x[s.ix] - x
    z = unit(torch.where(s.bisector, unit(u) + unit(v), u))
    ax = torch.where(s.bisector, unit(v), v)
    ax = unit(ax - (ax * z).sum(1, keepdim=True) * z)
    r = torch.stack([ax, torch.linalg.cross(z, ax), z], 2)
    dip = torch.einsum("nij,nj->ni", r, s.pole[:, 1:4])
    return s.pole[:, 0], dip, r @ s.pole[:, 4:].view(-1, 3, 3) @ r.transpose(1, 2)


def _pairs(x, box, cut):
    """Half pairs within cut (minimum image)."""
    n = len(x)
    rows = max(1, min(n, (1 << 26) // n))
    out = []
    for i0 in range(0, n, rows):
        r2 = 0.0
        for d in range(3):
            dx = x[None, i0:, d] - x[i0:i0 + rows, None, d]
            dx -= box[d] * torch.round(dx / box[d])
            r2 = r2 + dx * dx
        hit = (r2 <= cut * cut).triu(1).nonzero()
        out.append(hit + i0)
    return torch.cat(out).T.contiguous()


def _vector(x, box, i, k):
    r = x[k] - x[i]
    return r - box * torch.round((r / box).detach())


def _ewald(a, r2, order):
    """B0..B_order of the damped 1/r and the bare 1, 1, 3, 15, ... / r^(2l+1)."""
    r = r2.sqrt()
    b, bare = [torch.erfc(a * r) / r], [1.0 / r]
    ex, fac = torch.exp(-a * a * r2), 1.0 / (SQRT_PI * a)
    for q in range(1, order + 1):
        fac = fac * 2.0 * a * a
        b.append(((2 * q - 1) * b[-1] + fac * ex) / r2)
        bare.append((2 * q - 1) * bare[-1] / r2)
    return b, bare


def _thole(s, i, k, r):
    damp = torch.minimum(s.thole[i], s.thole[k]) * (r / (s.pdamp[i] * s.pdamp[k])) ** 3
    ex = torch.exp(-damp)
    return 1.0 - ex, 1.0 - (1.0 + damp) * ex, 1.0 - (1.0 + damp + 0.6 * damp * damp) * ex


def _direct_pairs(s, x, rp, i, k):
    """Permanent field at i from k and at k from i (the same for the d and p
    sets: pairs inside a molecule have scale 0 in both), and the mutual
    coefficients (scale 1)."""
    r = _vector(x, s.box, i, k)
    r2 = (r * r).sum(1)
    b, bare = _ewald(s.a, r2, 3)
    l3, l5, l7 = _thole(s, i, k, r2.sqrt())
    sc = (i // 3 != k // 3).to(r.dtype)
    f3, f5, f7 = (b[q] - (1.0 - sc * l) * bare[q] for q, l in ((1, l3), (2, l5), (3, l7)))
    dot = lambda u, v: (u * v).sum(1)

    def field(c, d, q, v):  # at a site from the moments at displacement v
        qv = torch.einsum("nij,nj->ni", q, v)
        rad = f3 * c - f5 * dot(d, v) + f7 * dot(qv, v)
        return -v * rad[:, None] - f3[:, None] * d + 2.0 * f5[:, None] * qv

    ei = field(rp[0][k], rp[1][k], rp[2][k], r)
    ek = field(rp[0][i], rp[1][i], rp[2][i], -r)
    return ei, ek, b[1] - (1.0 - l3) * bare[1], b[2] - (1.0 - l5) * bare[2], r


def _exact_dipoles(s, x, pairs):
    """(mu [n, 2, 3], Epol): conjugate gradients for both sets to 1e-13."""
    st, rp = _stencil(s, x), _rotate(s, x)
    e0 = -_gather_gradient(s, st, _convolve(s, _spread_poles(s, st, rp))) + s.term * rp[1]
    co = []
    for c in pairs.split(CHUNK, 1):
        ei, ek, c3, c5, r = _direct_pairs(s, x, rp, c[0], c[1])
        e0 = e0.index_add(0, c[0], ei).index_add(0, c[1], ek)
        co.append((c[0], c[1], c3[:, None], c5[:, None], r))

    def apply(v):
        h = v / s.alpha[:, None] + _gather_gradient(s, st, _convolve(s, _spread_dipoles(s, st, v))) - s.term * v
        for i, k, c3, c5, r in co:
            h.index_add_(0, i, c3 * v[k] - c5 * (r * v[k]).sum(1, keepdim=True) * r)
            h.index_add_(0, k, c3 * v[i] - c5 * (r * v[i]).sum(1, keepdim=True) * r)
        return h

    mu = s.alpha[:, None] * e0
    res = e0 - apply(mu)
    z = s.alpha[:, None] * res
    p, rz = z.clone(), (res * z).sum()
    stop = 1e-26 * (e0 * s.alpha[:, None] * e0).sum()
    for _ in range(80):
        if rz <= stop:
            break
        h = apply(p)
        al = rz / (p * h).sum()
        mu, res = mu + al * p, res - al * h
        z = s.alpha[:, None] * res
        new = (res * z).sum()
        p, rz = z + new / rz * p, new
    # the scales of a water box give the d and p sets the same field
    return mu, float(-0.5 * ELECTRIC * (mu * e0).sum())


def _backward(parts, x):
    """d(sum of the parts)/dx, each part a function of x differentiated alone."""
    g = torch.zeros_like(x)
    total = 0.0
    for f in parts:
        y = x.detach().clone().requires_grad_(True)
        e = f(y)
        g += torch.autograd.grad(e, y)[0]
        total += float(e.detach())
    return total, g


def _polarization_gradient(s, x, pairs, mu):
    """Gradient of L = -mu.E + mu.T.mu / 2 at fixed mu (stationary there)."""
    def recip(y):
        st, rp = _stencil(s, y), _rotate(s, y)
        gm = _spread_dipoles(s, st, mu)
        return ELECTRIC * ((gm * _convolve(s, _spread_poles(s, st, rp))).sum() + 0.5 * (gm * _convolve(s, gm)).sum()
                           - s.term * (mu * rp[1]).sum())

    def real(c):
        def f(y):
            i, k = c
            ei, ek, c3, c5, r = _direct_pairs(s, y, _rotate(s, y), i, k)
            mi, mk = mu[i], mu[k]
            e = -(mi * ei).sum() - (mk * ek).sum()
            return ELECTRIC * (e + (c3 * (mi * mk).sum(1) - c5 * (r * mi).sum(1) * (r * mk).sum(1)).sum())
        return f

    return _backward([recip] + [real(c) for c in pairs.split(CHUNK, 1)], x)[1]


def _multipole_energy(s, x, pairs):
    def recip(y):
        rp, st = _rotate(s, y), _stencil(s, y)
        g = _spread_poles(s, st, rp)
        t = 2.0 * s.a * s.a
        qq = (rp[2] * rp[2]).sum((1, 2))
        self_e = -s.a / SQRT_PI * (rp[0] ** 2 + t * ((rp[1] ** 2).sum(1) / 3.0 + 2.0 * t * qq / 5.0)).sum()
        return ELECTRIC * (0.5 * (g * _convolve(s, g)).sum() + self_e)

    def real(c):
        def f(y):
            i, k = c
            q, d, t = _rotate(s, y)
            r = _vector(y, s.box, i, k)
            b, bare = _ewald(s.a, (r * r).sum(1), 4)
            same = (i // 3 == k // 3).to(r.dtype)
            b = [u - same * v for u, v in zip(b, bare)]
            dot = lambda u, v: (u * v).sum(1)
            ci, di, ck, dk = q[i], d[i], q[k], d[k]
            qi, qk = (torch.einsum("nij,nj->ni", t[j], r) for j in (i, k))
            dir_, dkr, qir, qkr = dot(di, r), dot(dk, r), dot(qi, r), dot(qk, r)
            e = (ci * ck * b[0] + (ck * dir_ - ci * dkr + dot(di, dk)) * b[1]
                 + (ci * qkr + ck * qir - dir_ * dkr
                    + 2.0 * (dot(dk, qi) - dot(di, qk) + (t[i] * t[k]).sum((1, 2)))) * b[2]
                 + (dir_ * qkr - dkr * qir - 4.0 * dot(qi, qk)) * b[3] + qir * qkr * b[4])
            return ELECTRIC * e.sum()
        return f

    return _backward([recip] + [real(c) for c in pairs.split(CHUNK, 1)], x)


def _vdw_energy(s, x):
    v = s.vdw
    par, kred = _t(v["ired"], torch.int64), _t(v["kred"])[:, None]
    kred = torch.where(par[:, None] == torch.arange(s.n, device="cuda")[:, None], torch.ones_like(kred), kred)
    cls = _t(v["cls"], torch.int64)
    rmin, eps = _t(v["radmin"]).view(v["nclass"], -1), _t(v["eps"]).view(v["nclass"], -1)
    off, cut, gh, dh = v["vdwcut"], v["vdwtaper"], v["ghal"], v["dhal"]
    sites = lambda y: kred * (y - y[par]) + y[par]
    pairs = _pairs(sites(x), s.box, off)
    pairs = pairs[:, pairs[0] // 3 != pairs[1] // 3]

    def part(c):
        def f(y):
            i, k = c
            r = _vector(sites(y), s.box, i, k).norm(dim=1)
            rho = r / rmin[cls[i], cls[k]]
            e = eps[cls[i], cls[k]] * ((1 + dh) / (rho + dh)) ** 7 * ((1 + gh) / (rho ** 7 + gh) - 2.0)
            t = torch.clamp((r - cut) / (off - cut), min=0.0)
            return (e * (1.0 - t ** 3 * (10.0 - 15.0 * t + 6.0 * t * t))).sum()
        return f

    return _backward([part(c) for c in pairs.split(CHUNK, 1)], x)


def exact(case, seed):
    host = lambda t: t.cpu().numpy()
    if case["kind"] in ("solve", "batch"):
        boxes = _batch_boxes(case, seed) if case["kind"] == "batch" else [_box(case["nw"], seed)]
        mus, es = [], []
        for ws in boxes:
            s, x = _System(ws), _t(ws.positions())
            mu, e = _exact_dipoles(s, x, _pairs(x, s.box, s.cut))
            mus.append(host(mu))
            es.append(e)
        mu = np.concatenate(mus)
        return {"uind": mu, "uinp": mu, "epol": np.array(es) if case["kind"] == "batch" else es[0]}
    if 3 * case["nw"] > EXACT_ATOMS:
        return None
    ws = _box(case["nw"], seed)
    s = _System(ws)
    if case["kind"] == "step":
        out = []
        for p in _frames(ws, seed):
            x = _t(p)
            pairs = _pairs(x, s.box, s.cut)
            mu, e = _exact_dipoles(s, x, pairs)
            em, dem = _multipole_energy(s, x, pairs)
            ev, dev = _vdw_energy(s, x)
            out.append({"energies": np.array([e, em, ev]), "dep": host(_polarization_gradient(s, x, pairs, mu)),
                        "dem": host(dem), "dev": host(dev)})
            if case["virial"]:
                out[-1]["vir"] = None  # the reference's accumulation leaves terms of the strain derivative out
        return out
    water, params = _package().water, _package().params
    mass = water.masses(ws)
    vel = _t(water.maxwell_velocities(mass, 300.0, seed=seed))
    m = _t(mass)[:, None]
    x, energies = _t(ws.positions()), []

    def force(x):
        pairs = _pairs(x, s.box, s.cut)
        mu, e = _exact_dipoles(s, x, pairs)
        return e, -params.CONVERT * _polarization_gradient(s, x, pairs, mu) / m

    acc = force(x)[1]
    for _ in range(case["steps"]):
        vel = vel + 0.5 * DT * acc
        x = x + DT * vel
        e, acc = force(x)
        vel = vel + 0.5 * DT * acc
        kin = float(0.5 / params.CONVERT * (m * vel * vel).sum())
        energies.append([e, kin, e + kin])
    return {"pos": host(x), "vel": host(vel), "energies": np.array(energies)}
