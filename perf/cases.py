"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values.  Three kinds:

``evolve``    one lattice through ``Evolver.evolve(steps)`` with its analyser rows,
              then a snapshot of both time levels (``download_device``);
``ensemble``  many realisations of uneven sizes through ``Ensemble.evolve``, every
              member's rows, and one member's fields;
``transfer``  reference-layout fields into the evolver and back out
              (``upload_device`` / ``download_device``).

Initial data: links exp(i eps sigma.n) with eps ~ N(0, 0.1^2), phases N(0, 0.1^2),
doublets N(mean, 0.1^2) (mean 1 for SM, 0.7 for 2HDM, or a tanh wall along z), and
momenta of the size such fields reach after some steps (dt E with E ~ 0.3).
"""
import math
import random

import numpy as np
import torch

from gftevolver_b200 import GFT_MODEL_2HDM, GFT_MODEL_SM, Ensemble, Evolver, LatticeParams

DT, G, GP, GPP = 0.05, 0.65, 0.35, 0.5
MOMENTUM = 0.3
DOUBLE = ("fp64", "ref64")


def _evolve(name, model, form, nx, ny, nz, steps, log=10, family=0, fixed=0, wall=False):
    return {"name": name, "kind": "evolve", "model": model, "form": form, "nx": nx, "ny": ny, "nz": nz,
            "steps": steps, "log": log, "family": family, "fixed": fixed, "wall": wall}


def listed():
    return [
        # the headline workload: 256^3 SM in the mixed form, analysers every 10 steps
        _evolve("sm_mixed_256", "sm", "mixed", 256, 256, 256, 20),
        # the same physics at the size of a parameter scan
        _evolve("sm_mixed_128", "sm", "mixed", 128, 128, 128, 40),
        # a box chosen by physics, not by tiles: uneven edges, one of them odd
        _evolve("sm_mixed_ragged", "sm", "mixed", 150, 100, 75, 40),
        # the form for tight Gauss residuals, at the headline size
        _evolve("sm_fp64_256", "sm", "fp64", 256, 256, 256, 10),
        # the smallest benchmark configuration: launch-bound steps
        _evolve("sm_fp64_32", "sm", "fp64", 32, 32, 32, 100),
        # two doublets at the benchmark size, both forms
        _evolve("thdm_mixed_192", "2hdm", "mixed", 192, 192, 192, 20),
        _evolve("thdm_fp64_192", "2hdm", "fp64", 192, 192, 192, 10),
        # the reference's shipped configuration: 2HDM with the Higgs-family SU(2), 16^3
        _evolve("thdm_family_16", "2hdm", "mixed", 16, 16, 16, 20, family=2),
        # a bubble wall between Fixed z faces, with the family field: a production-size box
        _evolve("thdm_family_wall", "2hdm", "mixed", 96, 96, 192, 20, family=2, fixed=4, wall=True),
        # the parity form: the reference's own arithmetic and storage
        _evolve("sm_ref32_64", "sm", "ref32", 64, 64, 64, 10),
        # realisations of uneven sizes evolved together
        {"name": "ensemble_sm_32", "kind": "ensemble", "members": 32, "edges": "32,48,64,96", "steps": 20, "log": 10},
        # fields from and to a simulation that keeps them in the reference layout
        {"name": "transfer_sm_192", "kind": "transfer", "model": "sm", "form": "mixed", "nx": 192, "ny": 192,
         "nz": 192, "host": "f32"},
    ]


def draw(rng):
    def edge(lo, hi, any_size):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if any_size:
            return n
        step = rng.choice((8, 16, 32))
        return max(step, n // step * step)

    kind = rng.choice(("evolve",) * 8 + ("ensemble", "transfer"))
    if kind == "ensemble":
        edges = rng.choice(("32,48,64,96", "16,32,48", "32,64", "48,64,80"))
        return {"kind": kind, "members": rng.randint(6, 32), "edges": edges, "steps": 10 * rng.randint(1, 2), "log": 10}
    model = rng.choice(("sm", "2hdm"))
    form = rng.choice(("mixed", "mixed", "mixed", "fp64", "fp64", "ref32", "ref64"))
    any_size = rng.random() < 0.5
    hi = 72 if form in ("ref32", "ref64") else (140 if form == "fp64" else 200)
    nx, ny, nz = (edge(16, hi, any_size) for _ in range(3))
    if kind == "transfer":
        return {"kind": kind, "model": model, "form": form, "nx": nx, "ny": ny, "nz": nz,
                "host": rng.choice(("f32", "f64"))}
    family = rng.choice((0, 0, 0, 1, 2)) if model == "2hdm" else 0
    fixed = rng.choice((0, 0, 0, 0, 4, 2, 1, 5))
    # as many steps as keep the pass below the largest listed one
    most = min(100, max(2, int(1.5e8 / (nx * ny * nz) / (4 if form in ("ref32", "ref64") else 1))))
    return {"kind": kind, "model": model, "form": form, "nx": nx, "ny": ny, "nz": nz,
            "steps": rng.randint(max(1, most // 2), most), "log": rng.choice((0, 1, 5, 10, 10, 10)), "family": family,
            "fixed": fixed, "wall": model == "2hdm" and rng.random() < 0.3}


# ---- what a user's program has in hand -----------------------------------------------------------

def _params(c, nx, ny, nz):
    sm = c.get("model", "sm") == "sm"
    log = c.get("log", 0)
    common = dict(nx=nx, ny=ny, nz=nz, dt=DT, g=G, gp=GP, gpp=GPP, energy_every=log, gauss_every=log,
                  fixed_axes=c.get("fixed", 0), higgs_family=c.get("family", 0))
    if sm:
        return LatticeParams(model=GFT_MODEL_SM, lam=0.13, eta_sqr=1.0, **common)
    return LatticeParams(model=GFT_MODEL_2HDM, m1=0.5, m2=0.5, l1=0.065, l2=0.065, l3=0.2, m12r=0.2, l4p5=-0.1,
                         **common)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=g.device, dtype=torch.float32)


def _random_links(g, shape, dtype):
    """exp(i eps sigma.n) as unit quaternions [..., 4] of `dtype`, and the same after a small rotation."""
    n = _randn(g, *shape, 3).to(dtype)
    n = n / n.norm(dim=-1, keepdim=True).clamp_min(1e-6)
    eps = 0.1 * _randn(g, *shape, 1).to(dtype)
    past = torch.cat([torch.cos(eps), torch.sin(eps) * n], -1)
    v = DT * MOMENTUM * _randn(g, *shape, 3).to(dtype)
    u = torch.cat([torch.sqrt(1 - (v * v).sum(-1, keepdim=True)), v], -1)
    now = torch.stack(_qmul(u.unbind(-1), past.unbind(-1)), -1)
    return now, past


def _fields(c, nx, ny, nz, seed, dtype, device):
    """scalars[2, nx, ny, nz, nsc], vectors[2, nx, ny, nz, 3 dw]; slot 1 is "now", slot 0 "past" at time_iter 0."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    sm, family = c.get("model", "sm") == "sm", c.get("family", 0)
    nsc = 4 if sm else 8
    dw = {0: 5, 1: 6, 2: 9}[family]
    shape = (nx, ny, nz)
    sc = torch.empty((2, *shape, nsc), dtype=dtype, device=device)
    ve = torch.empty((2, *shape, 3 * dw), dtype=dtype, device=device)
    for k in range(nsc):
        f = 0.1 * _randn(g, *shape).to(dtype) + (1.0 if sm else 0.7)
        if c.get("wall"):
            f -= 0.7
            if k == 0:
                z = torch.arange(nz, device=device, dtype=dtype)
                f += 0.5 * (torch.tanh((z - nz / 4) / 5) - torch.tanh((z - 3 * nz / 4) / 5))
        sc[0, ..., k] = f
        sc[1, ..., k] = f + DT * MOMENTUM * _randn(g, *shape).to(dtype)
    for d in range(3):
        for at in ([0, 5] if family == 1 else [0]):
            th = 0.1 * _randn(g, *shape).to(dtype)
            ve[0, ..., dw * d + at] = th
            ve[1, ..., dw * d + at] = th + DT * MOMENTUM * _randn(g, *shape).to(dtype)
        for at in ([1, 5] if family == 2 else [1]):
            now, past = _random_links(g, shape, dtype)
            ve[0, ..., dw * d + at:dw * d + at + 4] = past
            ve[1, ..., dw * d + at:dw * d + at + 4] = now
    return sc, ve


def _edges(case):
    pick = random.Random(case["members"])
    edges = [int(e) for e in case["edges"].split(",")]
    return [tuple(pick.choice(edges) for _ in range(3)) for _ in range(case["members"])]


def prepare(case, seed):
    if case["kind"] == "ensemble":
        sizes = _edges(case)
        ens = Ensemble([_params(case, *s) for s in sizes])
        for m, s in enumerate(sizes):
            sc, ve = _fields(case, *s, seed * 1000 + m, torch.float32, "cuda")
            ens.upload(m, sc.cpu().numpy(), ve.cpu().numpy(), 0)
        small = min(range(len(sizes)), key=lambda m: (sizes[m][0] * sizes[m][1] * sizes[m][2], m))
        return {"case": case, "ens": ens, "show": small}
    size = (case["nx"], case["ny"], case["nz"])
    ev = Evolver(_params(case, *size), form=case["form"])
    f64 = case["host"] == "f64" if case["kind"] == "transfer" else case["form"] in DOUBLE
    sc, ve = _fields(case, *size, seed, torch.float64 if f64 else torch.float32, "cuda")
    torch.cuda.synchronize()
    state = {"case": case, "ev": ev, "f64": f64, "out": (torch.empty_like(sc), torch.empty_like(ve))}
    if case["kind"] == "transfer":
        state["in"] = (sc, ve)
    else:
        ev.upload_device(sc.data_ptr(), ve.data_ptr(), f64, 0)
    return state


# ---- one pass --------------------------------------------------------------------------------------

ENERGIES = ("energy", "potential", "gradient", "kinetic", "magnetic", "electric", "plaq_su2", "plaq_u1", "phi_sq")


def _table(rows, dtype):
    """The analyser rows as one array per quantity."""
    out = {k: np.array([r[k] for r in rows], dtype) for k in ENERGIES}
    for k in ("gauss_int", "gauss_max"):
        out[k] = np.array([r[k] for r in rows], dtype)
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        rows = state["ens"].evolve(case["steps"])
        sc, ve = state["ens"].download(state["show"])
        return {"rows": _table([r for member in rows for r in member], np.float32), "scalars": sc, "vectors": ve}
    ev, (sc, ve) = state["ev"], state["out"]
    if case["kind"] == "transfer":
        a, b = state["in"]
        ev.upload_device(a.data_ptr(), b.data_ptr(), state["f64"], 0)
        ev.download_device(sc.data_ptr(), ve.data_ptr(), state["f64"])
        return {"scalars": sc, "vectors": ve}
    rows = ev.evolve(case["steps"])
    ev.download_device(sc.data_ptr(), ve.data_ptr(), state["f64"])
    return {"rows": _table(rows, np.float64 if state["f64"] else np.float32) if rows else {}, "scalars": sc,
            "vectors": ve}


# ---- what a pass cannot do without -----------------------------------------------------------------

def _words(case):
    """Stored words of one site of one level."""
    return (19 if case.get("model", "sm") == "sm" else 23) + {0: 0, 1: 3, 2: 12}[case.get("family", 0)]


def _site_flops(case):
    """Multiplies and adds of one site's update (staples, transports, currents, series)."""
    return (2300 if case.get("model", "sm") == "sm" else 3000) + {0: 0, 1: 400, 2: 1600}[case.get("family", 0)]


def work(case):
    """Every step reads both levels and writes one; a logging step's Gauss constraint reads both once more;
    a snapshot reads and writes both."""
    if case["kind"] == "ensemble":
        sites = sum(x * y * z for x, y, z in _edges(case))
        size, steps, shown = 4, case["steps"], min(x * y * z for x, y, z in _edges(case))
    else:
        sites = shown = case["nx"] * case["ny"] * case["nz"]
        size, steps = (8 if case["form"] in DOUBLE else 4), case.get("steps", 0)
    w = _words(case)
    host = {"f32": 4, "f64": 8}.get(case.get("host"), size)
    if case["kind"] == "transfer":
        return {"bytes": 4.0 * w * sites * (size + host), "flops": 0.0}
    logs = len([t for t in range(steps) if case["log"] and t % case["log"] == 0])
    return {"bytes": float(sites * w * size * (3 * steps + 2 * logs) + 4 * w * size * shown),
            "flops": float(sites * _site_flops(case) * steps)}


# ---- the same in 64 bits ---------------------------------------------------------------------------

def _qmul(a, b):
    """The product (a0 b0 - a.b, a0 b + b0 a - a x b)."""
    return (a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3],
            a[0] * b[1] + a[1] * b[0] - a[2] * b[3] + a[3] * b[2],
            a[0] * b[2] + a[2] * b[0] - a[3] * b[1] + a[1] * b[3],
            a[0] * b[3] + a[3] * b[0] - a[1] * b[2] + a[2] * b[1])


def _conj(a):
    return (a[0], -a[1], -a[2], -a[3])


def _at(f, axis, by):
    """The field at x + by e_axis."""
    if isinstance(f, (tuple, list)):
        return tuple(_at(c, axis, by) for c in f)
    return torch.roll(f, -by, axis)


def _act(u, h):
    """The 4x4 real action of a link quaternion on a doublet."""
    w, x, y, z = u
    return (w * h[0] - z * h[1] + y * h[2] - x * h[3], z * h[0] + w * h[1] + x * h[2] + y * h[3],
            -y * h[0] - x * h[1] + w * h[2] + z * h[3], x * h[0] - y * h[1] - z * h[2] + w * h[3])


def _phase(f, th, sign):
    c, s = torch.cos(th), sign * torch.sin(th)
    return (c * f[0] - s * f[1], c * f[1] + s * f[0], c * f[2] - s * f[3], c * f[3] + s * f[2])


class _Exact:
    """One lattice in 64 bits: the leapfrog step and the analysers, all sites at once."""

    def __init__(self, case, sc, ve, fixed_mask):
        self.family = case.get("family", 0)
        self.nd = 1 if case.get("model", "sm") == "sm" else 2
        self.levels = [self._split(sc[t], ve[t]) for t in (0, 1)]
        self.mask = fixed_mask  # 1 where evolved, None: everywhere

    def _split(self, sc, ve):
        dw = {0: 5, 1: 6, 2: 9}[self.family]
        word = lambda k: ve[..., k].double().contiguous()  # noqa: E731
        lv = {"th": [word(dw * d) for d in range(3)],
              "q": [tuple(word(dw * d + 1 + k) for k in range(4)) for d in range(3)],
              "ph": [tuple(sc[..., 4 * b + k].double().contiguous() for k in range(4)) for b in range(self.nd)]}
        if self.family == 1:
            lv["hth"] = [word(dw * d + 5) for d in range(3)]
        if self.family == 2:
            lv["hq"] = [tuple(word(dw * d + 5 + k) for k in range(4)) for d in range(3)]
        return lv

    def join(self, t):
        lv = self.levels[t]
        per = []
        for d in range(3):
            per += [lv["th"][d], *lv["q"][d]]
            if self.family == 1:
                per.append(lv["hth"][d])
            if self.family == 2:
                per += lv["hq"][d]
        return torch.stack([k for b in lv["ph"] for k in b], -1), torch.stack(per, -1)

    @staticmethod
    def _loops(u):
        """Per direction, sum over planes of vec(P1) - vec(P2); and the traces of the three plaquettes."""
        force, trace = [], []
        for i in range(3):
            f = [0.0, 0.0, 0.0]
            for j in range(3):
                if i == j:
                    continue
                ui, uj = u[i], u[j]
                p1 = _qmul(_qmul(_qmul(_conj(_at(uj, i, 1)), _at(ui, j, 1)), uj), _conj(ui))
                back = _at(uj, j, -1)
                p2 = _qmul(_qmul(_qmul(ui, back), _conj(_at(ui, j, -1))), _conj(_at(_at(uj, i, 1), j, -1)))
                f = [f[k] + p1[k + 1] - p2[k + 1] for k in range(3)]
                if i < j:
                    trace.append(p1[0] / torch.sqrt(sum(c * c for c in p1)))
            force.append(f)
        return force, trace

    @staticmethod
    def _phases(th):
        force, angle = [], []
        for i in range(3):
            f = 0.0
            for j in range(3):
                if i == j:
                    continue
                up = th[i] + _at(th[j], i, 1) - _at(th[i], j, 1) - th[j]
                lo = th[i] + _at(th[j], j, -1) - _at(th[i], j, -1) - _at(_at(th[j], i, 1), j, -1)
                f = f - torch.sin(up) - torch.sin(lo)
                if i < j:
                    angle.append(up)
            force.append(f)
        return force, angle

    def _family(self, t, sign, lv, d, back):
        """The family link of direction d (at x, or at x - d) on the transported doublets."""
        if self.family == 1:
            h = _at(lv["hth"][d], d, -1) if back else lv["hth"][d]
            return [_phase(t[0], h, sign), _phase(t[1], h, -sign)]
        if self.family == 2:
            h = _at(lv["hq"][d], d, -1) if back else lv["hq"][d]
            h = h if sign > 0 else _conj(h)
            lo, hi = _act(h, (*t[0][:2], *t[1][:2])), _act(h, (*t[0][2:], *t[1][2:]))
            return [(lo[0], lo[1], hi[0], hi[1]), (lo[2], lo[3], hi[2], hi[3])]
        return t

    def _sum(self, v):
        return float((v if self.mask is None else v * self.mask).sum())

    def step(self, ti, energy, gauss):
        now, old = self.levels[(ti + 1) % 2], self.levels[ti % 2]
        dt2, nd, fam = DT * DT, self.nd, self.family
        forces, traces = self._loops(now["q"])
        yforce, angles = self._phases(now["th"])
        if fam == 1:
            hforce, hangles = self._phases(now["hth"])
        elif fam == 2:
            hforce, htraces = self._loops(now["hq"])
        lap = [tuple(-6.0 * c for c in now["ph"][b]) for b in range(nd)]
        cur, hcur, grad = [], [], 0.0
        for a in range(3):
            ua, ta = now["q"][a], now["th"][a]
            fp = [_at(now["ph"][b], a, 1) for b in range(nd)]
            tm = [_act(_at(ua, a, -1), _phase(_at(now["ph"][b], a, -1), _at(ta, a, -1), 1)) for b in range(nd)]
            tp = [_act(_conj(ua), _phase(fp[b], ta, -1)) for b in range(nd)]
            t = [_act(ua, _phase(now["ph"][b], ta, 1)) for b in range(nd)]
            tm, t = self._family(tm, 1, now, a, True), self._family(t, 1, now, a, False)
            tp = self._family(tp, -1, now, a, False)
            lap = [tuple(lap[b][k] + tm[b][k] + tp[b][k] for k in range(4)) for b in range(nd)]
            j = [0.0] * 4
            for b in range(nd):
                u, f = t[b], fp[b]
                j[0] = j[0] + 0.25 * (u[0] * f[1] - u[1] * f[0] + u[2] * f[3] - u[3] * f[2])
                j[1] = j[1] + 0.25 * (u[0] * f[3] - u[1] * f[2] + u[2] * f[1] - u[3] * f[0])
                j[2] = j[2] + 0.25 * (-u[0] * f[2] - u[1] * f[3] + u[2] * f[0] + u[3] * f[1])
                j[3] = j[3] + 0.25 * (u[0] * f[1] - u[1] * f[0] - u[2] * f[3] + u[3] * f[2])
                if energy:
                    grad = grad + 0.5 * sum((f[k] - u[k]) ** 2 for k in range(4))
            cur.append(j)
            if fam:
                hcur.append(self._family_current([*t[0], *t[1]], [*fp[0], *fp[1]]))
            del tm, tp, t, fp
        pot, pot_e = self._potential(now["ph"])
        row = {}
        if energy:
            kin = sum((a - b) ** 2 for p, q in zip(now["ph"], old["ph"]) for a, b in zip(p, q)) * (0.5 / dt2)
            inv = {"g": 1 / G ** 2, "gp": 1 / GP ** 2, "gpp": 1 / GPP ** 2}
            mag = sum(4 * inv["g"] * (1 - t) for t in traces) + sum(4 * inv["gp"] * (1 - torch.cos(x)) for x in angles)
            if fam == 1:
                mag = mag + sum(4 * inv["gpp"] * (1 - torch.cos(x)) for x in hangles)
            elif fam == 2:
                mag = mag + sum(4 * inv["gpp"] * (1 - t) for t in htraces)
            ele = 0.0
            for d in range(3):
                ele = ele + 4 / dt2 * inv["g"] * (1 - self._turn(now["q"][d], old["q"][d]))
                ele = ele + 4 / dt2 * inv["gp"] * (1 - torch.cos(now["th"][d] - old["th"][d]))
                if fam == 1:
                    ele = ele + 4 / dt2 * inv["gpp"] * (1 - torch.cos(now["hth"][d] - old["hth"][d]))
                elif fam == 2:
                    ele = ele + 4 / dt2 * inv["gpp"] * (1 - self._turn(now["hq"][d], old["hq"][d]))
            n = float(pot_e.numel() if self.mask is None else self.mask.expand_as(pot_e).sum())
            row.update(potential=self._sum(pot_e), gradient=self._sum(grad), kinetic=self._sum(kin),
                       magnetic=self._sum(mag), electric=self._sum(ele), plaq_su2=self._sum(sum(traces)) / (3 * n),
                       plaq_u1=self._sum(sum(torch.cos(x) for x in angles)) / (3 * n),
                       phi_sq=self._sum(sum(c * c for p in now["ph"] for c in p)) / n)
            row["energy"] = sum(row[k] for k in ENERGIES[1:6])
        new = {"ph": [tuple(2 * c - p + dt2 * (a - v) for c, p, a, v in zip(*x))
                      for x in zip(now["ph"], old["ph"], lap, pot)]}
        g2 = (GP * GP, G * G)
        new["th"] = [now["th"][d] + torch.asin(torch.sin(now["th"][d] - old["th"][d]) +
                                               dt2 * (yforce[d] + g2[0] * cur[d][0])) for d in range(3)]
        new["q"] = [self._advance(now["q"][d], old["q"][d],
                                  [dt2 * (forces[d][k] + g2[1] * cur[d][k + 1]) for k in range(3)]) for d in range(3)]
        if fam == 1:
            new["hth"] = [now["hth"][d] + torch.asin(torch.sin(now["hth"][d] - old["hth"][d]) +
                                                     dt2 * (hforce[d] + GPP ** 2 * hcur[d][0])) for d in range(3)]
        elif fam == 2:
            new["hq"] = [self._advance(now["hq"][d], old["hq"][d],
                                       [dt2 * (hforce[d][k] + GPP ** 2 * hcur[d][k]) for k in range(3)])
                         for d in range(3)]
        if self.mask is not None:  # sites on Fixed faces keep what they hold
            keep = self.mask > 0
            pick = lambda a, b: (tuple(torch.where(keep, x, y) for x, y in zip(a, b)) if isinstance(a, tuple)  # noqa: E731
                                 else torch.where(keep, a, b))
            new = {k: [pick(a, b) for a, b in zip(new[k], old[k])] for k in new}
        self.levels[ti % 2] = new
        if gauss:
            row["gauss_int"], row["gauss_max"] = self._gauss(now, new)
        return row

    @staticmethod
    def _turn(a, b):
        p = _qmul(a, _conj(b))
        return p[0] / torch.sqrt(sum(c * c for c in p))

    @staticmethod
    def _advance(now, old, add):
        e = _qmul(now, _conj(old))
        r = [e[k + 1] + add[k] for k in range(3)]
        u = (torch.sqrt(1 - r[0] ** 2 - r[1] ** 2 - r[2] ** 2), *r)
        new = _qmul(u, now)
        norm = torch.sqrt(sum(c * c for c in new))
        return tuple(c / norm for c in new)

    def _family_current(self, t, n):
        h = [0.0, 0.0, 0.0]
        for i in (0, 2):
            own = t[i] * n[i + 1] - t[i + 1] * n[i] - t[i + 4] * n[i + 5] + t[i + 5] * n[i + 4]
            if self.family == 1:
                h[0] = h[0] + 0.25 * own
            else:
                h[0] = h[0] + 0.25 * (t[i] * n[i + 5] - t[i + 1] * n[i + 4] + t[i + 4] * n[i + 1] - t[i + 5] * n[i])
                h[1] = h[1] + 0.25 * (-t[i] * n[i + 4] - t[i + 1] * n[i + 5] + t[i + 4] * n[i] + t[i + 5] * n[i + 1])
                h[2] = h[2] + 0.25 * own
        return h

    def _potential(self, ph):
        if self.nd == 1:
            f = ph[0]
            s = sum(c * c for c in f) - 1.0
            return [tuple(0.13 * s * c for c in f)], 0.25 * 0.13 * s * s
        m1, m2, l1, l2, l3, m12r, l45 = 0.5, 0.5, 0.065, 0.065, 0.2, 0.2, -0.1
        a, b = ph
        s1, s2, dot = sum(c * c for c in a), sum(c * c for c in b), sum(x * y for x, y in zip(a, b))
        c1 = -2 * m1 + 4 * l1 * s1 + 2 * l3 * s2
        c2 = -2 * m2 + 4 * l2 * s2 + 2 * l3 * s1
        mix = -m12r + 2 * l45 * dot
        v = -m1 * s1 - m2 * s2 + l1 * s1 * s1 + l2 * s2 * s2 + l3 * s1 * s2 - m12r * dot + l45 * dot * dot
        return [tuple(c1 * x + mix * y for x, y in zip(a, b)), tuple(c2 * y + mix * x for x, y in zip(a, b))], v

    def _gauss(self, now, new):
        el = [0.0] * 4
        for d in range(3):
            turn = torch.sin(new["th"][d] - now["th"][d])
            el[0] = el[0] + turn - _at(turn, d, -1)
            here = _qmul(_conj(now["q"][d]), new["q"][d])
            back = _at(_qmul(new["q"][d], _conj(now["q"][d])), d, -1)
            for k in range(1, 4):
                el[k] = el[k] + here[k] - back[k]
        rho = [0.0] * 4
        for p, q in zip(now["ph"], new["ph"]):
            rho[0] = rho[0] + 0.25 * (p[0] * q[1] - p[1] * q[0] + p[2] * q[3] - p[3] * q[2])
            rho[1] = rho[1] + 0.25 * (p[0] * q[3] - p[1] * q[2] + p[2] * q[1] - p[3] * q[0])
            rho[2] = rho[2] + 0.25 * (-p[0] * q[2] - p[1] * q[3] + p[2] * q[0] + p[3] * q[1])
            rho[3] = rho[3] + 0.25 * (p[0] * q[1] - p[1] * q[0] - p[2] * q[3] + p[3] * q[2])
        off = [el[k] - (GP ** 2 if k == 0 else G ** 2) * rho[k] for k in range(4)]
        if self.family:
            he = [0.0] * 3
            for d in range(3):
                if self.family == 1:
                    turn = torch.sin(new["hth"][d] - now["hth"][d])
                    he[0] = he[0] + turn - _at(turn, d, -1)
                else:
                    here = _qmul(_conj(now["hq"][d]), new["hq"][d])
                    back = _at(_qmul(new["hq"][d], _conj(now["hq"][d])), d, -1)
                    for k in range(3):
                        he[k] = he[k] + here[k + 1] - back[k + 1]
            hr = self._family_current([*now["ph"][0], *now["ph"][1]], [*new["ph"][0], *new["ph"][1]])
            off += [he[k] - GPP ** 2 * hr[k] for k in range(1 if self.family == 1 else 3)]
        off = [v.abs() if self.mask is None else v.abs() * self.mask for v in off]
        return [float(v.sum()) for v in off], [float(v.max()) for v in off]


def _exact_lattice(case, size, sc, ve):
    mask = None
    if case.get("fixed"):
        mask = torch.ones(size, dtype=torch.float64, device=sc.device)
        for a in range(3):
            if case["fixed"] >> a & 1:
                mask.select(a, 0).zero_()
                mask.select(a, size[a] - 1).zero_()
    ex, log, rows = _Exact(case, sc, ve, mask), case.get("log", 0), []
    for ti in range(case["steps"]):
        logs = bool(log) and ti % log == 0
        row = ex.step(ti, logs, logs)
        if logs:
            rows.append(row)
    return ex, rows


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "ensemble":
        sizes = _edges(case)
        small = min(range(len(sizes)), key=lambda m: (sizes[m][0] * sizes[m][1] * sizes[m][2], m))
        rows = []
        for m, s in enumerate(sizes):
            ex, got = _exact_lattice(case, s, *_fields(case, *s, seed * 1000 + m, torch.float32, device))
            rows += got
            if m == small:
                shown = ex
    else:
        size = (case["nx"], case["ny"], case["nz"])
        f64 = case["host"] == "f64" if case["kind"] == "transfer" else case["form"] in DOUBLE
        sc, ve = _fields(case, *size, seed, torch.float64 if f64 else torch.float32, device)
        if case["kind"] == "transfer":
            return {"scalars": sc.double(), "vectors": ve.double()}
        shown, rows = _exact_lattice(case, size, sc, ve)
    lv = [shown.join(t) for t in (0, 1)]
    return {"rows": _table(rows, np.float64) if rows else {}, "scalars": torch.stack([a for a, _ in lv]),
            "vectors": torch.stack([b for _, b in lv])}
