"""The work that is timed: molecular dynamics, minimisation, single evaluations
and served jobs over atoms and 8-node elements, through ``cac_b200.api``.

Systems are the FCC slabs of ``cac_b200.gen`` (``[element layers][atomic
layers][element layers]``; 162 nx ny atoms per atomic layer, 2 nx ny elements
per element layer and region), built here on the GPU from a seed: every
coordinate displaced by up to 0.01 a, Maxwell-Boltzmann velocities, x-strain.
Potentials are the two of the repository's workloads: LJ (0.4093 eV, 2.338 A,
cutoff 5.5 A) and the analytic EAM tabulated to 10,000 points (cutoff 5.0 A),
taken smoothly to zero at the cutoff as published EAM tables are; skin 1.0 A,
lists rebuilt every 10 steps, 1 fs.

``exact`` evaluates the same model in 64 bits with plain torch and numpy.  The
mixed form integrates in 64 bits and forms forces from 32-bit pair sums: its
runs hand over atom positions in 64 bits, and forces, velocities, energies
and the coarse elements' nodes (which the forces drive apart soonest) in 32.
"""
import dataclasses
import math
import random

import numpy as np
import torch

from cac_b200 import api, gen

LATTICE = 3.615
MASS = 63.546
BOLTZ = 8.617343e-5
MVV2E = 1.0364269e-4
LJ = (0.4093, 2.338, 5.5)
SKIN = 1.0
EVERY = 10
DT = 0.001
SIDE = 9                      # lattice sites per element edge
CELL = SIDE ** 3              # lattice sites per element
NODE_WEIGHT = CELL / 8.0
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
LANGEVIN = (300.0, 300.0, 0.1, 48271)   # start, stop (K), damping (ps), seed
ERATE = 0.5                             # x strain rate of the tension tests (1/ps)


def listed():
    eam, lj = dict(pair="eam"), dict(pair="lj")
    return [
        # an outer program (a driver, a fitting loop) hands over new positions of a
        # small system and reads energies, forces and virials: the smallest call
        dict(name="point_tiny_lj_fp64", kind="point", form="fp64", **lj, nx=3, ny=1, le=1, la=3, temp=50.0, strain=0.0,
             host=True),
        # the small LJ slab a user validates with: latency and launches
        dict(name="run100_small_lj_fp64", kind="run", form="fp64", **lj, nx=3, ny=1, le=18, la=9, temp=10.0, strain=0.0,
             steps=100, fix="none"),
        # a mid-sized ragged LJ run in the mixed form
        dict(name="run25_mid_lj_mixed", kind="run", form="mixed", **lj, nx=5, ny=3, le=7, la=33, temp=100.0, strain=0.0,
             steps=25, fix="none"),
        # one evaluation with every tally (a thermo or dump step) after a restart
        dict(name="point_eam_fp64", kind="point", form="fp64", **eam, nx=8, ny=5, le=32, la=42, temp=300.0, strain=0.0,
             host=False),
        # thermostatted EAM run
        dict(name="nvt20_eam_fp64", kind="run", form="fp64", **eam, nx=7, ny=5, le=23, la=39, temp=300.0, strain=0.0,
             steps=20, fix="langevin"),
        # the million-atom EAM run in FP64
        dict(name="run20_1m_eam_fp64", kind="run", form="fp64", **eam, nx=8, ny=5, le=125, la=162, temp=300.0,
             strain=0.0, steps=20, fix="none"),
        # the four-million-atom strained EAM run in the mixed form: the largest
        dict(name="run20_4m_eam_mixed", kind="run", form="mixed", **eam, nx=20, ny=10, le=125, la=129, temp=300.0,
             strain=0.03, steps=20, fix="none"),
        # a tension test: the box stretched every step
        dict(name="tension20_eam_mixed", kind="run", form="mixed", **eam, nx=7, ny=3, le=9, la=57, temp=300.0, strain=0.0,
             steps=20, fix="deform"),
        # independent replicas of uneven size as one batch
        dict(name="batch64_eam_mixed", kind="run", form="mixed", **eam, replicas=64, atoms=64000, elements=2000,
             temp=300.0, strain=0.02, steps=20, fix="none"),
        # a small batch in FP64
        dict(name="batch12_lj_fp64", kind="run", form="fp64", **lj, replicas=12, atoms=16000, elements=400, temp=100.0,
             strain=0.01, steps=30, fix="none"),
        # relaxation by FIRE
        dict(name="fire50_eam_fp64", kind="fire", form="fp64", **eam, nx=6, ny=4, le=15, la=21, temp=0.0, strain=0.01,
             steps=50),
        # served jobs: minimisations and short runs of different sizes, submitted together
        dict(name="serve10_lj_mixed", kind="serve", form="mixed", **lj, jobs=10, atoms=50000, elements=1200, temp=50.0,
             strain=0.02, steps=25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "batch", "point", "fire", "serve"])
    c = dict(form=rng.choice(["fp64", "mixed"]), pair=rng.choice(["eam", "eam", "lj"]))
    c["temp"] = round(rng.uniform(10.0, 400.0), 1)
    c["strain"] = round(rng.uniform(0.0, 0.04), 4)
    if kind == "serve":
        return dict(c, kind="serve", pair="lj", jobs=rng.randint(3, 12), atoms=_log(rng, 4000, 50000),
                    elements=_log(rng, 60, 1200), steps=rng.randint(15, 25))
    if kind == "batch":
        return dict(c, kind="run", replicas=_log(rng, 3, 64), atoms=_log(rng, 4000, 64000),
                    elements=_log(rng, 60, 2000), steps=rng.randint(12, 22), fix="none")
    nx, ny = rng.randint(3, 11), rng.randint(1, 7)
    la = 3 * max(1, min(42, _log(rng, 600, 1200000) // (486 * nx * ny)))
    le = max(1, min(60, _log(rng, 12, 20000) // (4 * nx * ny)))
    c = dict(c, nx=nx, ny=ny, le=le, la=la)
    # the dynamics of coarse elements is not stable over long runs, and 32-bit
    # pair sums drift apart sooner than 64-bit ones
    most = 45 if c["form"] == "fp64" else 22
    if kind == "point":
        return dict(c, kind="point", host=rng.random() < 0.4)
    if kind == "fire":
        return dict(c, kind="fire", temp=0.0, steps=rng.randint(12, most))
    return dict(c, kind="run", steps=rng.randint(12, most), fix=rng.choice(["none", "none", "langevin", "deform"]))


# ------------------------------------------------------------------- inputs


def _replica_shape(atoms, elements):
    """Slab dimensions with about these counts (as ``cac_b200.gen.replica``)."""
    nxy = max(2, min(atoms // 486, elements // 4))
    nx = max(2, int(math.ceil(math.sqrt(nxy))))
    ny = max(1, int(round(nxy / nx)))
    la = max(3, 3 * int(round(atoms / (162 * nx * ny) / 3.0)))
    return nx, ny, max(1, int(round(elements / (4.0 * nx * ny)))), la


def _shapes(case):
    """(nx, ny, le, la) of each system of a case: one, or replicas and jobs
    whose sizes spread log-uniformly up to the case's largest."""
    n = case.get("replicas") or case.get("jobs")
    if not n:
        return [(case["nx"], case["ny"], case["le"], case["la"])]
    rng = random.Random(1000 * n + 7)
    a0, e0 = (2000, 50) if case.get("replicas") else (1000, 20)
    return [_replica_shape(_log(rng, a0, max(a0 + 1, case["atoms"])), _log(rng, e0, max(e0 + 1, case["elements"])))
            for _ in range(n)]


def _counts(case):
    return [(162 * nx * ny * la, 4 * nx * ny * le) for nx, ny, le, la in _shapes(case)]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _slab(shape, temp, strain, g):
    """One slab on the device: the geometry of ``cac_b200.gen.build_slab``."""
    nx, ny, le, la = shape
    dev = _device()
    f8 = dict(dtype=torch.float64, device=dev)
    b = LATTICE / math.sqrt(2.0)
    A = torch.tensor([[b, 0.0, 0.0], [0.5 * b, math.sqrt(0.75) * b, 0.0],
                      [0.5 * b, math.sqrt(1.0 / 12.0) * b, math.sqrt(2.0 / 3.0) * b]], **f8)
    dz = b * math.sqrt(2.0 / 3.0)
    L = torch.tensor([SIDE * b * nx, SIDE * math.sqrt(3.0) * b * ny, (2 * SIDE * le + la) * dz], **f8)
    origin = torch.tensor([0.25 * b, 0.125 * b * math.sqrt(3.0), 0.5 * dz], **f8)

    def points(ni, nj, layers, step):
        i = torch.arange(ni, **f8)[None, :, None]
        j = torch.arange(nj, **f8)[None, None, :]
        k = torch.tensor(layers, **f8)[:, None, None]
        p = origin + step * (i[..., None] * A[0] + j[..., None] * A[1]) + k[..., None] * A[2]
        p = p.expand(len(layers), ni, nj, 3).reshape(-1, 3).clone()
        p[:, :2] -= torch.floor(p[:, :2] / L[:2]) * L[:2]
        return p

    x = points(SIDE * nx, 2 * SIDE * ny, list(range(SIDE * le, SIDE * le + la)), 1)
    starts = [SIDE * m for m in range(le)] + [SIDE * le + la + SIDE * m for m in range(le)]
    corner = (SIDE - 1) * torch.tensor(CORNERS, **f8) @ A
    nodex = points(nx, 2 * ny, starts, SIDE)[:, None, :] + corner[None]
    jitter = lambda a: a + (2 * torch.rand(a.shape, generator=g, **f8) - 1) * (0.01 * LATTICE)  # noqa: E731
    x, nodex = jitter(x), jitter(nodex)
    sigma = math.sqrt(BOLTZ * temp / (MASS * MVV2E))
    v = sigma * torch.randn(x.shape, generator=g, **f8)
    nodev = sigma * torch.randn(nodex.shape, generator=g, **f8)
    x[:, 0] *= 1.0 + strain
    nodex[..., 0] *= 1.0 + strain
    L[0] *= 1.0 + strain
    x -= torch.floor(x / L) * L
    nodex -= (torch.floor(nodex.mean(1) / L) * L)[:, None, :]
    return dict(lo=torch.zeros(3, **f8), hi=L, x=x, v=v, nodex=nodex, nodev=nodev)


def _systems(case, seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    n = case.get("replicas") or case.get("jobs") or 1
    # replicas and jobs differ in temperature and strain as well
    return [_slab(s, case["temp"] * (0.5 + k / n), case["strain"] * (k + 1) / n, g) for k, s in
            enumerate(_shapes(case))]


def _host(s):
    c = lambda t: t.cpu().numpy()  # noqa: E731
    return gen.System(boxlo=c(s["lo"]), boxhi=c(s["hi"]), x=c(s["x"]), v=c(s["v"]), nodex=c(s["nodex"]),
                      nodev=c(s["nodev"]), mass=MASS, lattice_a=LATTICE)


def _eam_tables():
    p = gen.EamParams()
    frho, rhor, z2r = p.tables()
    s = ((p.cut - np.arange(p.nr) * p.dr).clip(0.0) / 0.5) ** 4
    rhor, z2r = rhor * s / (1.0 + s), z2r * s / (1.0 + s)
    return dict(nrho=p.nrho, drho=p.drho, nr=p.nr, dr=p.dr, cut=p.cut, mass=p.mass, frho=frho, rhor=rhor, z2r=z2r)


@dataclasses.dataclass
class State:
    case: dict
    engine: object = None
    host: list = None
    server: object = None


def _form(case):
    return api.MIXED if case["form"] == "mixed" else api.FP64


def _set_pair(target, case):
    if case["pair"] == "lj":
        target.pair_lj(*LJ)
    else:
        target.pair_eam(_eam_tables())
    target.neighbor(SKIN, EVERY)


def prepare(case, seed):
    systems = [_host(s) for s in _systems(case, seed)]
    if case["kind"] == "serve":
        srv = api.Server(workers=4, precision=_form(case))
        _set_pair(srv, case)
        srv.start()
        return State(case, host=systems, server=srv)
    eng = api.Engine()
    eng.set_precision(_form(case))
    if case.get("replicas"):
        eng.upload_batch(systems)
    else:
        eng.upload(systems[0])
    _set_pair(eng, case)
    if case.get("fix") == "langevin":
        eng.langevin(*LANGEVIN)
    if case.get("fix") == "deform":
        eng.deform(1, x=("erate", ERATE))
    eng.snapshot()
    keep = case.get("host") or case.get("fix") == "deform"
    return State(case, engine=eng, host=systems if keep else None)


# ------------------------------------------------------------------ one pass


def _single(t):
    return t.astype(np.float32) if isinstance(t, np.ndarray) else t.float()


def _arrays(eng, case, names):
    """Device arrays of the context, converted on its own stream.  They share
    its memory, so each keeps the context."""
    out = {}
    with torch.cuda.stream(torch.cuda.ExternalStream(eng.stream)):
        for n in names:
            t = eng.device_array(n)
            if n == "x":
                t = t[:, :3]
            single = case["form"] == "mixed" and not (n == "x" and case["kind"] == "run")
            out[n] = _single(t) if single else t
            out[n].context = eng
    return out


def _scalar(case, v):
    return torch.tensor(v, dtype=torch.float32 if case["form"] == "mixed" else torch.float64)


def run(state):
    case, eng = state.case, state.engine
    if case["kind"] == "run":
        eng.restore()
        if case["fix"] == "langevin":
            eng.langevin_stream(1)
        if case["fix"] == "deform":
            eng.set_box(state.host[0].boxlo, state.host[0].boxhi)
        eng.run_nve(case["steps"], DT)
        return _arrays(eng, case, ("x", "v", "f", "nodex", "nodev", "nodef"))
    if case["kind"] == "point":
        if case["host"]:
            eng.set_state(x=state.host[0].x, nodex=state.host[0].nodex)
            eng.build_lists()
        else:
            eng.restore()
        eng.compute(api.ENERGY_GLOBAL | api.ENERGY_ATOM, api.VIRIAL_GLOBAL | api.VIRIAL_ATOM)
        out = _arrays(eng, case, ("f", "nodef", "eatom", "enode", "vatom", "vnode"))
        ev = eng.energy(peratom=False)
        out["energy"] = _scalar(case, ev["energy"])
        out["virial"] = _scalar(case, ev["virial"])
        return out
    if case["kind"] == "fire":
        eng.restore()
        code, iterations, energy, fnorm = eng.minimize_fire(maxiter=case["steps"], ftol=1e-6, dt=DT)
        out = _arrays(eng, case, ("x", "nodex", "f", "nodef"))
        out["energy"], out["fnorm"] = _scalar(case, energy), _scalar(case, fnorm)
        out["stop"] = (code, iterations)
        return out
    # a served stream: everything submitted, then each result taken
    srv, jobs = state.server, []
    for k, s in enumerate(state.host):
        kind = api.JOB_NVE if _is_run(k) else api.JOB_FIRE
        jobs.append(srv.submit(s, kind, case["steps"], DT, 0.0, 1e-6))
    out = []
    for job in jobs:
        if srv.wait(job) != 0:
            raise RuntimeError("a served job failed: " + srv.last_error())
        x, v, nodex, nodev, energy, iterations, code, _ = srv.result(job)
        srv.release(job)
        if case["form"] == "mixed":
            x, nodex = _single(x), _single(nodex)
        out.append(dict(x=x, nodex=nodex, energy=_scalar(case, energy), stop=(code, iterations)))
    return out


def _is_run(k):
    """Three jobs in ten are short runs, the others minimisations."""
    return k % 10 in (2, 5, 8)


def work(case):
    """State in and out once; distances within cutoff + skin at each list
    build, pair terms within the cutoff at each force evaluation."""
    atoms = sum(a for a, _ in _counts(case))
    elements = sum(e for _, e in _counts(case))
    sites = atoms + 8 * elements
    volume = LATTICE ** 3 / 4.0
    near = lambda r: 4.0 / 3.0 * math.pi * r ** 3 / volume  # noqa: E731
    cut, per_pair = (LJ[2], 24) if case["pair"] == "lj" else (5.0, 52)
    steps = case.get("steps", 0)
    pair = sites * near(cut) * per_pair * (steps + 1)
    build = sites * near(cut + SKIN) * 9 * (1 + steps // EVERY)
    state = 24 * sites
    moved = state * (2 if case["kind"] == "point" else 5)
    if case["kind"] == "point":
        moved += 8 * 7 * sites
    return dict(bytes=float(moved), flops=float(pair + build))


# ------------------------------------------------- the same model in 64 bits


def _spline(values, delta):
    """Cubic value coefficients per interval of a tabulated function, with
    fourth-order slopes at the knots; (coefficients [n, 4], 1/delta)."""
    f = np.asarray(values, dtype=np.float64)
    n = f.size
    s = np.empty(n)
    s[0], s[1] = f[1] - f[0], 0.5 * (f[2] - f[0])
    s[n - 2], s[n - 1] = 0.5 * (f[n - 1] - f[n - 3]), f[n - 1] - f[n - 2]
    s[2:n - 2] = ((f[:n - 4] - f[4:]) + 8.0 * (f[3:n - 1] - f[1:n - 3])) / 12.0
    c = np.zeros((n, 4))
    c[:, 0], c[:, 1] = f, s
    d = f[1:] - f[:-1]
    c[:-1, 2] = 3.0 * d - 2.0 * s[:-1] - s[1:]
    c[:-1, 3] = s[:-1] + s[1:] - 2.0 * d
    return torch.tensor(c, device=_device()), 1.0 / delta


def _lookup(table, r):
    """(value, derivative) of a tabulated function."""
    c, rd = table
    p = r * rd
    m = p.long().clamp(0, c.shape[0] - 2)
    p = (p - m).clamp(max=1.0)
    k = c[m]
    return (((k[:, 3] * p + k[:, 2]) * p + k[:, 1]) * p + k[:, 0],
            ((3.0 * k[:, 3] * p + 2.0 * k[:, 2]) * p + k[:, 1]) * rd)


class Model:
    """Atoms and elements of one or several periodic boxes: forces on atoms
    and nodes from atoms and interpolated lattice sites, velocity Verlet."""

    CHUNK = 48_000_000   # pairs, or candidates, at a time

    def __init__(self, systems, pair):
        dev = _device()
        cat = lambda k: torch.cat([s[k] for s in systems])  # noqa: E731
        self.lo = torch.stack([s["lo"] for s in systems])
        self.hi = torch.stack([s["hi"] for s in systems])
        self.x, self.v, self.nodex, self.nodev = (cat(k).clone() for k in ("x", "v", "nodex", "nodev"))
        self.na, self.ne = self.x.shape[0], self.nodex.shape[0]
        rep = lambda k: torch.cat([torch.full((s[k].shape[0],), i, device=dev) for i, s in enumerate(systems)])  # noqa: E731
        self.arep, self.erep = rep("x"), rep("nodex")
        self.irep = torch.cat([self.arep, self.erep.repeat_interleave(8)])
        self.pair = pair
        self.cut = LJ[2] if pair == "lj" else gen.EamParams().cut
        if pair == "eam":
            t = _eam_tables()
            self.f_table = _spline(t["rhor"], t["dr"])
            self.z_table = _spline(t["z2r"], t["dr"])
            self.e_table = _spline(t["frho"], t["drho"])
        u = torch.arange(CELL, device=dev)
        n = torch.stack([u // 81, u // 9 % 9, u % 9], 1).double() / 8.0
        c = torch.tensor(CORNERS, dtype=torch.float64, device=dev)
        self.shape = (c[None] * n[:, None] + (1 - c[None]) * (1 - n[:, None])).prod(2)     # [729, 8]
        self.minv = torch.where(c[:, None] == c[None], 4.0, -2.0).prod(2).double()
        self.iscale = torch.cat([torch.ones(self.na, device=dev), torch.full((8 * self.ne,), NODE_WEIGHT, device=dev)])

    def wrap(self):
        lo, hi = self.lo[self.arep], self.hi[self.arep]
        L = hi - lo
        self.x += torch.where(self.x < lo, L, 0.0)
        self.x -= torch.where(self.x >= hi, L, 0.0)
        lo, hi = self.lo[self.erep], self.hi[self.erep]
        L = hi - lo
        c = self.nodex.mean(1)
        self.nodex += (torch.where(c < lo, L, 0.0) - torch.where(c >= hi, L, 0.0))[:, None]

    def sites(self):
        """Positions of the lattice sites in use, from the nodes."""
        p = torch.zeros(self.su.numel(), 3, dtype=torch.float64, device=self.x.device)
        for k in range(8):
            p += self.shape[self.su, k][:, None] * self.nodex[self.se, k]
        return p

    def build(self):
        """Pairs (i-site, j-site, image) within cutoff + skin."""
        self.wrap()
        dev, rc = self.x.device, self.cut + SKIN
        L = self.hi - self.lo
        nc = torch.floor(L / rc).long()
        base = torch.cat([torch.zeros(1, dtype=torch.long, device=dev), nc.prod(1).cumsum(0)])
        xi = torch.cat([self.x, self.nodex.reshape(-1, 3)])
        self.se = torch.arange(self.ne, device=dev).repeat_interleave(CELL)
        self.su = torch.arange(CELL, device=dev).repeat(self.ne)
        sites = self.sites()
        xj = torch.cat([self.x, sites])
        jrep = torch.cat([self.arep, self.erep[self.se]])

        def place(p, rep):
            t = torch.floor((p - self.lo[rep]) / L[rep])
            w = p - t * L[rep]
            c = torch.minimum(((w - self.lo[rep]) * (nc[rep] / L[rep])).long().clamp(min=0), nc[rep] - 1)
            return w, -t.to(torch.int8), c

        wj, tj, cj = place(xj, jrep)
        key = base[jrep] + (cj[:, 2] * nc[jrep, 1] + cj[:, 1]) * nc[jrep, 0] + cj[:, 0]
        key, order = key.sort()
        first = torch.searchsorted(key, torch.arange(int(base[-1]) + 1, device=dev))
        wj, tj = wj[order], tj[order]
        wi, ti, ci = place(xi, self.irep)
        got = []
        n_i = xi.shape[0]
        per = max(1, self.CHUNK // 4)
        for oz in (-1, 0, 1):
            for oy in (-1, 0, 1):
                for ox in (-1, 0, 1):
                    o = torch.tensor([ox, oy, oz], device=dev)
                    for a in range(0, n_i, per // 8):
                        i = torch.arange(a, min(n_i, a + per // 8), device=dev)
                        r = self.irep[i]
                        c = ci[i] + o
                        W = torch.div(c, nc[r], rounding_mode="floor")
                        c -= W * nc[r]
                        k = base[r] + (c[:, 2] * nc[r, 1] + c[:, 1]) * nc[r, 0] + c[:, 0]
                        count = first[k + 1] - first[k]
                        ii = torch.arange(i.numel(), device=dev).repeat_interleave(count)
                        if not ii.numel():
                            continue
                        jj = torch.arange(ii.numel(), device=dev) - (count.cumsum(0) - count)[ii] + first[k][ii]
                        shift = W.double() * L[r]
                        d = wi[i][ii] - (wj[jj] + shift[ii])
                        d = (d * d).sum(1)
                        ok = (d <= rc * rc) & (d > 1e-6)
                        ii, jj = ii[ok], jj[ok]
                        S = tj[jj] + W.to(torch.int8)[ii] - ti[i][ii]
                        got.append((ii + a, order[jj], S))
        self.pi, self.pj, self.ps = (torch.cat(t) for t in zip(*got))
        # the lattice sites that are neighbours
        used = torch.zeros(xj.shape[0], dtype=torch.bool, device=dev)
        used[self.pj] = True
        used[:self.na] = True
        rank = used.cumsum(0) - 1
        self.pj = rank[self.pj].int()
        self.pi = self.pi.int()
        keep = used[self.na:]
        self.se, self.su = self.se[keep], self.su[keep]

    def _terms(self, xj):
        """Per chunk of pairs within the cutoff: i, j, separation, distance."""
        xi = torch.cat([self.x, self.nodex.reshape(-1, 3)])
        L = self.hi - self.lo
        one = L.shape[0] == 1
        for a in range(0, self.pi.numel(), self.CHUNK):
            i, j = self.pi[a:a + self.CHUNK].long(), self.pj[a:a + self.CHUNK].long()
            d = xi[i] - xj[j] - self.ps[a:a + self.CHUNK] * (L if one else L[self.irep[i]])
            rsq = (d * d).sum(1)
            ok = rsq < self.cut * self.cut
            yield i[ok], j[ok], d[ok], rsq[ok].sqrt()

    def forces(self, tally=False, energy_weight=NODE_WEIGHT):
        dev = self.x.device
        n_i = self.na + 8 * self.ne
        zero = lambda *s: torch.zeros(*s, dtype=torch.float64, device=dev)  # noqa: E731
        xj = torch.cat([self.x, self.sites()])
        fi, e, vir, emb = zero(n_i, 3), zero(n_i), zero(n_i, 6), zero(n_i)
        if self.pair == "eam":
            rho = zero(n_i)
            for i, j, d, r in self._terms(xj):
                rho.index_add_(0, i, _lookup(self.f_table, r)[0])
            nrho = rho[self.na:].view(-1, 8)
            srho = zero(self.su.numel())
            for k in range(8):
                srho += self.shape[self.su, k] * nrho[self.se, k]
            emb, fp = _lookup(self.e_table, rho)
            fpj = torch.cat([fp[:self.na], _lookup(self.e_table, srho)[1]])
        else:
            eps, sig, _ = LJ
            c12, c6 = 4 * eps * sig ** 12, 4 * eps * sig ** 6
        for i, j, d, r in self._terms(xj):
            if self.pair == "eam":
                df = _lookup(self.f_table, r)[1]
                z, dz = _lookup(self.z_table, r)
                phi = z / r
                pull = -((fp[i] + fpj[j]) * df + dz / r - phi / r) / r
            else:
                r6 = r ** -6
                phi = r6 * (c12 * r6 - c6)
                pull = r6 * (12 * c12 * r6 - 6 * c6) / (r * r)
            fi.index_add_(0, i, d * pull[:, None])
            if tally:
                e.index_add_(0, i, phi)
                vir.index_add_(0, i, d[:, [0, 1, 2, 0, 0, 1]] * d[:, [0, 1, 2, 1, 2, 2]] * pull[:, None])
        self.f = fi[:self.na]
        self.nodef = torch.einsum("ab,ebd->ead", self.minv, fi[self.na:].view(-1, 8, 3) / 8.0)
        if tally:
            w = self.iscale.double()
            we = torch.cat([torch.ones(self.na, device=dev), torch.full((8 * self.ne,), energy_weight, device=dev)]).double()
            self.esite, self.vsite = 0.5 * e + emb, 0.5 * vir
            self.energy = float((we * self.esite).sum())
            self.virial = (w[:, None] * self.vsite).sum(0)

    def kick(self):
        dtfm = 0.5 * DT / MVV2E / MASS
        self.v += dtfm * self.f
        self.nodev += dtfm * self.nodef

    def run(self, steps, fix):
        self.build()
        self.forces()
        noise = Noise(self, steps) if fix == "langevin" else None
        if noise:
            noise.add()
        lo0, hi0 = self.lo.clone(), self.hi.clone()
        for s in range(1, steps + 1):
            self.kick()
            self.x += DT * self.v
            self.nodex += DT * self.nodev
            if s % EVERY == 0:
                self.build()
            self.forces()
            if noise:
                noise.add()
            self.kick()
            if fix == "deform":
                grow = 0.5 * ERATE * DT * s * (hi0[:, 0] - lo0[:, 0])
                lo, hi = self.lo.clone(), self.hi.clone()
                lo[:, 0], hi[:, 0] = lo0[:, 0] - grow, hi0[:, 0] + grow
                for p, r in ((self.x, self.arep), (self.nodex.view(-1, 3), self.irep[self.na:])):
                    p.copy_((p - self.lo[r]) / (self.hi - self.lo)[r] * (hi - lo)[r] + lo[r])
                self.lo, self.hi = lo, hi

    def fire(self, maxiter, ftol):
        """FIRE 2.0 (Guenole et al. 2020) from rest; (stop code, iterations,
        energy, squared force norm).  While minimising, an EAM node weighs one
        site in the energy."""
        weight = 1.0 if self.pair == "eam" else NODE_WEIGHT
        self.v.zero_()
        self.nodev.zero_()
        self.build()
        self.forces(True, weight)
        dt = dtv = DT
        alpha, back, since, it = 0.25, 0.0, 0, 0
        while True:
            # the sites are wrapped whenever lists are rebuilt
            f = torch.cat([self.f, self.nodef.reshape(-1, 3)])
            v = torch.cat([self.v, self.nodev.reshape(-1, 3)])
            fnorm = float((f * f).sum(1).max())
            stop = 3 if it > 0 and fnorm < ftol * ftol else 0 if it >= maxiter else None
            if stop is not None:
                self.wrap()
                return stop, it, self.energy, fnorm
            it += 1
            power = float((v * f).sum())
            if power > 0:
                if it - since > 20:
                    dt, alpha = min(dt * 1.1, 10 * DT), alpha * 0.99
            else:
                since = it
                if it >= 20:
                    alpha = 0.25
                    if dt * 0.5 >= 0.02 * DT:
                        dt *= 0.5
            fastest = float(v.abs().max()) if power > 0 else dt / MVV2E / MASS * float(f.abs().max())
            back = 0.0 if power > 0 else 0.5 * dtv
            dtv = min(dt, 0.1 / fastest) if fastest > 0 else dt
            ff = float((f * f).sum())
            mix = alpha * math.sqrt(float((v * v).sum()) / ff) if ff > 1e-20 else 0.0
            x = torch.cat([self.x, self.nodex.view(-1, 3)])
            if not power > 0:
                x = x - back * v
                v = torch.zeros_like(v)
            v = v + dtv / MVV2E / MASS * f
            if power > 0:
                v = (1.0 - alpha) * v + mix * f
            x = x + dtv * v
            self.x, self.v = x[:self.na].clone(), v[:self.na].clone()
            self.nodex, self.nodev = x[self.na:].view(-1, 8, 3).clone(), v[self.na:].view(-1, 8, 3).clone()
            if it % EVERY == 0:
                self.build()
            self.forces(True, weight)


class Noise:
    """Langevin drag and random force from the RANMAR generator (Marsaglia,
    Zaman and Tsang; F. James 1990), drawn over atoms, then nodes."""

    def __init__(self, model, steps):
        self.m = model
        t, _, damp, seed = LANGEVIN
        ij, kl = divmod(seed - 1, 30082)
        i, j, k, l = ij // 177 % 177 + 2, ij % 177 + 2, kl // 169 % 178 + 1, kl % 169
        u = []
        for _ in range(97):
            s = 0
            for bit in range(24):
                i, j, k = j, k, i * j % 179 * k % 179
                l = (53 * l + 1) % 169
                if l * k % 64 >= 32:
                    s |= 1 << (23 - bit)
            u.append(s)
        self.n = 3 * model.na + 24 * model.ne
        total = 1 + self.n * (steps + 1)
        y = np.zeros(97 + total + 33, dtype=np.int64)
        y[:97] = u[::-1]
        for a in range(97, 97 + total, 33):
            y[a:a + 33] = (y[a - 97:a - 64] - y[a - 33:a]) & 0xFFFFFF
        m = np.arange(1, total + 1, dtype=np.int64)
        c = (362436 - m * 7654321 % 16777213) % 16777213
        self.u = ((y[97:97 + total] - c) & 0xFFFFFF)[1:] / 16777216.0
        self.at = 0
        ftm2v = 1.0 / MVV2E
        self.g1 = -MASS / damp / ftm2v
        self.g2 = math.sqrt(MASS) * math.sqrt(24.0 * BOLTZ / damp / DT / MVV2E) / ftm2v * math.sqrt(t)

    def add(self):
        m = self.m
        u = torch.from_numpy(self.u[self.at:self.at + self.n]).to(m.x.device) - 0.5
        self.at += self.n
        m.f = m.f + self.g1 * m.v + self.g2 * u[:3 * m.na].view(-1, 3)
        m.nodef = m.nodef + self.g1 * m.nodev + self.g2 / math.sqrt(NODE_WEIGHT) * u[3 * m.na:].view(-1, 8, 3)


def exact(case, seed):
    systems = _systems(case, seed)
    host = lambda t: t.cpu()  # noqa: E731
    flat = lambda t: host(t.reshape(-1, 3))  # noqa: E731
    if case["kind"] == "serve":
        out = []
        for k, s in enumerate(systems):
            m = Model([s], case["pair"])
            if _is_run(k):
                m.run(case["steps"], "none")
                m.forces(True)
                stop, energy = (0, case["steps"]), m.energy
            else:
                code, it, energy, _ = m.fire(case["steps"], 1e-6)
                stop = (code, it)
                m.forces(True)
            out.append(dict(x=host(m.x), nodex=host(m.nodex), energy=torch.tensor(energy, dtype=torch.float64), stop=stop))
        return out
    m = Model(systems, case["pair"])
    if case["kind"] == "run":
        m.run(case["steps"], case["fix"])
        return dict(x=host(m.x), v=host(m.v), f=host(m.f), nodex=flat(m.nodex), nodev=flat(m.nodev), nodef=flat(m.nodef))
    if case["kind"] == "point":
        m.build()
        m.forces(True)
        return dict(f=host(m.f), nodef=flat(m.nodef), eatom=host(m.esite[:m.na]), enode=host(m.esite[m.na:]),
                    vatom=host(m.vsite[:m.na]), vnode=host(m.vsite[m.na:]),
                    energy=torch.tensor(m.energy, dtype=torch.float64), virial=host(m.virial))
    code, it, energy, fnorm = m.fire(case["steps"], 1e-6)
    return dict(x=host(m.x), nodex=flat(m.nodex), f=host(m.f), nodef=flat(m.nodef), energy=torch.tensor(energy, dtype=torch.float64),
                fnorm=torch.tensor(fnorm, dtype=torch.float64), stop=(code, it))
