"""Workloads of the explicit update and of the steps around it, timed through the public API.

Each case is a plain dict; prepare() makes a user's inputs on the GPU from a seed, run() takes one
pass through vidyut_b200.api, work() states the bytes and operations the pass cannot do without and
exact() restates it in 64-bit torch.  Kinds of case:

  update   one explicit step of one box (api.explicit_update_all), the call a time loop makes per box
  percall  the same step through the one-loop-at-a-time entry points a host drops in for the
           reference's own loops (reaction source, face fluxes and dsdt per species, Joule heating)
  coupled  one step of a time loop with the potential solve: potential and fields, time scales, update
  species  the implicit diffusion solve of one species on a box that is the whole domain
  batch    many uneven independent boxes stepped together (api.Batch): load, step, read back
  serve    requests on host memory through the continuous-batching server (api.Server)

Boxes, mechanisms and value ranges are those of vidyut_b200.inputs and bench.py; the fields are made
on the GPU because a 128^3 state takes numpy half a minute.
"""
import math
import random

import torch

from vidyut_b200 import _abi as abi
from vidyut_b200 import api, inputs
from vidyut_b200 import mechanism as mm

S = inputs.BASE_SEED
MECHS = {  # name: (species, reactions); the mechanisms of the repository's configurations
    "argon4": (4, 10),
    "synth8": (8, 40),
    "synth12": (12, 60),
    "synth24": (24, 150),
}
DENS = {"argon4": (1e14, 1e18), "synth8": (1e10, 1e18), "synth12": (1e10, 1e18), "synth24": (1e8, 1e22)}
PREC = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED}
DX = 1e-5
G = 3

_mechs = {}
_loaded = None


def mechanism(name):
    """The mechanism, loaded into the library when it is not the one loaded last (a program
    loads its mechanism once)."""
    global _loaded
    if name not in _mechs:
        seed = {"argon4": S + 1, "synth8": S + 21, "synth12": S + 31, "synth24": S + 11}[name]
        _mechs[name] = mm.argon(10, seed) if name == "argon4" else mm.synthetic(*MECHS[name], seed)
    if _loaded != name:
        api.mech_init(_mechs[name])
        _loaded = name
    return _mechs[name]


# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # the smallest call of a time loop: a 1-D column, where latency and launches count
        dict(name="update_1d", kind="update", mech="synth8", nx=300, ny=1, nz=1, order=5, weno=3, precision="fp64",
             evolve=1, rates=0),
        # the 2-D argon configuration, one box of an AMReX level, with dsdt and rxn wanted by the host
        dict(name="update_2d_argon", kind="update", mech="argon4", nx=256, ny=256, nz=1, order=5, weno=3,
             precision="fp64", evolve=0, rates=1),
        # an ordinary 2-D discharge of odd extents in a mixed-precision time loop
        dict(name="update_2d_mixed", kind="update", mech="synth8", nx=467, ny=509, nz=1, order=5, weno=3,
             precision="mixed", evolve=1, rates=0),
        # the benchmark's headline: 128^3, 24 species, 150 reactions, plain FP64 ...
        dict(name="update_3d", kind="update", mech="synth24", nx=128, ny=128, nz=128, order=5, weno=3,
             precision="fp64", evolve=0, rates=0),
        # ... and in mixed precision
        dict(name="update_3d_mixed", kind="update", mech="synth24", nx=128, ny=128, nz=128, order=5, weno=3,
             precision="mixed", evolve=0, rates=0),
        # a ragged 3-D box with the second-order scheme
        dict(name="update_3d_ragged", kind="update", mech="synth12", nx=97, ny=61, nz=45, order=2, weno=3,
             precision="fp64", evolve=1, rates=1),
        # the per-call drop-in on a 2-D box: one flux call per species and direction
        dict(name="percall_2d", kind="percall", mech="synth8", nx=256, ny=256, nz=1, order=5, weno=3),
        # the same on a 3-D box of an AMReX level
        dict(name="percall_3d", kind="percall", mech="synth12", nx=64, ny=64, nz=64, order=5, weno=1),
        # one step of the large single case: potential solve, time scales, mixed update
        dict(name="coupled_3d", kind="coupled", mech="synth12", nx=256, ny=256, nz=256, precision="mixed"),
        # the semi-implicit step's electron solve
        dict(name="species_2d", kind="species", mech="argon4", nx=512, ny=512, nz=1, spec="electron", walls="hneu"),
        # the batched workload: uneven 2-D boxes, 20 steps each
        dict(name="batch_2d", kind="batch", mech="synth8", boxes=16, lo=64, hi=512, steps=20, precision="mixed",
             ones=0),
        # a burst of 1-D and 2-D requests to the server
        dict(name="serve", kind="serve", mech="synth8", boxes=6, lo=256, hi=512, steps=100, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, dim, cells_lo, cells_hi, step=1):
    """Extents with a product log-uniform in [cells_lo, cells_hi] and sides within a factor of two."""
    side = math.exp(rng.uniform(math.log(cells_lo), math.log(cells_hi)) / dim)
    n = [max(16, int(round(side * math.exp(rng.uniform(-0.3, 0.3)) / step)) * step) if d < dim else 1 for d in range(3)]
    while n[0] * n[1] * n[2] > cells_hi:
        n[n.index(max(n))] -= step
    return n


def draw(rng: random.Random):
    """One more case of the ranges above: every kind, scheme, precision and mechanism, odd extents
    (multiples of 8 where a multigrid solves, as an AMReX level's boxes are)."""
    kind = rng.choice(["update", "update", "update", "percall", "coupled", "species", "batch", "serve"])
    if kind == "update":
        dim = rng.choice([1, 2, 2, 3, 3])
        mech = rng.choice(["synth8"] if dim == 1 else ["argon4", "synth8", "synth12"] if dim == 2 else
                          ["synth8", "synth12", "synth24"])
        n = _sides(rng, dim, *{1: (256, 4096), 2: (64 * 64, 1024 * 1024), 3: (24**3, 2_000_000)}[dim])
        order = rng.choice([5, 5, 5, 2, 1])
        return dict(kind=kind, mech=mech, nx=n[0], ny=n[1], nz=n[2], order=order, weno=rng.choice([1, 2, 3, 3]),
                    precision=rng.choice(["fp64", "mixed"]), evolve=rng.choice([0, 1]),
                    rates=0 if mech == "synth24" else rng.choice([0, 1]))
    if kind == "percall":
        dim = rng.choice([2, 3])
        n = _sides(rng, dim, *{2: (64 * 64, 512 * 512), 3: (24**3, 96**3)}[dim])
        return dict(kind=kind, mech=rng.choice(["argon4", "synth8", "synth12"]), nx=n[0], ny=n[1], nz=n[2],
                    order=rng.choice([5, 5, 2, 1]), weno=rng.choice([1, 2, 3]))
    if kind == "coupled":
        dim = rng.choice([2, 3])
        n = _sides(rng, dim, *{2: (128 * 128, 1024 * 1024), 3: (48**3, 192**3)}[dim], step=8)
        return dict(kind=kind, mech=rng.choice(["synth8", "synth12"]), nx=n[0], ny=n[1], nz=n[2],
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "species":
        dim = rng.choice([2, 3])
        n = _sides(rng, dim, *{2: (64 * 64, 1024 * 1024), 3: (32**3, 128**3)}[dim], step=8)
        return dict(kind=kind, mech="argon4", nx=n[0], ny=n[1], nz=n[2], spec=rng.choice(["electron", "ion", "energy"]),
                    walls=rng.choice(["hneu", "ihneu"]))
    if kind == "batch":
        return dict(kind=kind, mech="synth8", boxes=rng.randint(4, 16), lo=64, hi=_log(rng, 128, 512), steps=20,
                    precision=rng.choice(["fp64", "mixed", "mixed"]), ones=rng.choice([0, 1, 2]))
    return dict(kind=kind, mech="synth8", boxes=rng.randint(3, 6), lo=256, hi=_log(rng, 300, 512),
                steps=_log(rng, 50, 100), precision=rng.choice(["fp64", "mixed"]))


# ---------------------------------------------------------------------------
# inputs


def _dim(c):
    return 3 if c["nz"] > 1 else 2 if c["ny"] > 1 else 1


def _ghosts(a, dim, n, comps=None):
    """First-order extrapolation into the face-adjacent ghosts and, direction by direction, the corners."""
    for d in range(dim):
        ax = 3 - d
        for q in range(1, G + 1):
            a.narrow(ax, G - q, 1).copy_(a.narrow(ax, G, 1))
            a.narrow(ax, G + n[d] - 1 + q, 1).copy_(a.narrow(ax, G + n[d] - 1, 1))


def _valid(a, dim, n):
    for d in range(dim):
        a = a.narrow(a.dim() - 1 - d, G, n[d])
    return a


def _smooth(gen, rnd, n, dim):
    """A sum of six random cosines with a uniform marginal, in [0, 1)."""
    ax = [(torch.arange(n[d], device="cuda", dtype=torch.float64) + 0.5) / n[d] for d in range(3)]
    g = torch.zeros((n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
    var = 0.0
    for _ in range(6):
        k = [rnd.randint(-2, 2) if d < dim else 0 for d in range(3)]
        if not any(k):
            k[0] = 1
        a, ph = rnd.gauss(0.0, 1.0), rnd.uniform(0.0, 2 * math.pi)
        xy = 2 * math.pi * (k[0] * ax[0][None, :] + k[1] * ax[1][:, None]) + ph
        z = 2 * math.pi * k[2] * ax[2][:, None, None]
        g += a * (torch.cos(xy)[None] * torch.cos(z) - torch.sin(xy)[None] * torch.sin(z))
        var += 0.5 * a * a
    return torch.special.ndtr(g / math.sqrt(max(var, 1e-30))).clamp_(0.0, 1.0 - 1e-15)


class Box:
    """One box as a user's program holds it: the ghosted state, the face fields and the parameters."""

    def __init__(self, mech, dim, n, seed, *, dens, blob=False, voltage=1000.0, bg=2.4e25, te=(0.3, 10.0), ramp=False,
                 faces=True, **prm):
        rnd = random.Random(seed)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        ns = mech.ns
        self.mech, self.dim, self.n = mech, dim, tuple(n)
        gv = [G if d < dim else 0 for d in range(3)]
        st = torch.zeros((mech.nvar, n[2] + 2 * gv[2], n[1] + 2 * gv[1], n[0] + 2 * gv[0]), dtype=torch.float64,
                         device="cuda")
        v = _valid(st, dim, n)
        x = [(torch.arange(n[d], device="cuda", dtype=torch.float64) + 0.5) / n[d] for d in range(3)]
        if blob:  # the argon configuration: a Gaussian electron blob, ions matching, the rest at the floor
            peak = 10.0 ** rnd.uniform(14.0, 18.0)
            r2 = 0.0
            for d in range(dim):
                r2 = r2 + (((x[d] - rnd.uniform(0.35, 0.65)) * 8.0) ** 2).reshape([-1 if e == 2 - d else 1 for e in range(3)])
            ne = 1e10 + peak * torch.exp(-0.5 * r2)
        for s in range(ns):
            if s in mech.bg_species:
                v[s] = bg
            elif blob:
                v[s] = ne if (s == mech.e_id or mech.charge[s] > 0) else 1e10
            else:
                lo, hi = math.log10(dens[0]), math.log10(dens[1])
                v[s] = torch.pow(10.0, lo + (hi - lo) * _smooth(gen, rnd, n, dim))
        v[ns + 1] = (te[0] + (te[1] - te[0]) * torch.rand(v[0].shape, generator=gen, dtype=torch.float64,
                                                          device="cuda")) * EV
        if ramp:
            v[ns + 2] = (voltage * (1.0 - x[0]))[None, None, :]
        else:
            xi = 2.0 * torch.rand(v[0].shape, generator=gen, dtype=torch.float64, device="cuda") - 1.0
            v[ns + 2] = voltage * x[0][None, None, :] * (1.0 + 0.05 * xi)
        _ghosts(st, dim, n)
        if not ramp:  # cell field by centred differences, reduced field
            pot = st[ns + 2]
            e2 = 0.0
            for d in range(dim):
                p = _valid_but(pot, dim, n, d)
                ax = 2 - d
                e = -(p.narrow(ax, G + 1, n[d]) - p.narrow(ax, G - 1, n[d])) / (2 * DX)
                v[ns + 3 + d] = e
                e2 = e2 + e * e
            v[ns + 9] = torch.sqrt(e2) / v[:ns].sum(0) / 1e-21
            _ghosts(st, dim, n)
        st[ns] = 1.5 * st[mech.e_id] * K_B * st[ns + 1]
        self.state = st
        self.ef, self.gn = [], []
        for d in range(3):
            shp = [1, n[2] + (d == 2 and d < dim), n[1] + (d == 1 and d < dim), n[0] + (d == 0)]
            if not faces or d >= dim:
                self.ef.append(torch.zeros(shp, dtype=torch.float64, device="cuda"))
                self.gn.append(torch.zeros(shp, dtype=torch.float64, device="cuda"))
                continue
            for comp, sign, out in ((ns + 2, -1.0, self.ef), (mech.e_id, 1.0, self.gn)):
                p = _valid_but(st[comp], dim, n, d)
                f = sign * (p.narrow(2 - d, G, n[d] + 1) - p.narrow(2 - d, G - 1, n[d] + 1)) / DX
                out.append(f.reshape(shp).contiguous())
        self.params = dict(dim=dim, dx=(DX,) * 3, n=self.n, bg_mask=mech.bg_mask(), **prm)
        self.case = inputs.BoxCase(mech=mech, dim=dim, n=self.n, ghost=G, dx=(DX,) * 3, state=None, efield=[], gradne=[],
                                   params=self.params, seed=seed)
        self.dc = api.DeviceCase(self.case, st, self.ef, self.gn)
        self.prm = self.case.vd_params()

    def hosted(self):
        """The case with its arrays on the host, as Batch.add and Server.submit take them."""
        c = self.case
        c.state = self.state.cpu().numpy()
        c.efield = [t.cpu().numpy() for t in self.ef]
        c.gradne = [t.cpu().numpy() for t in self.gn]
        return c


def _valid_but(a, dim, n, d):
    """The valid range in every direction but d (3-d array)."""
    for e in range(dim):
        if e != d:
            a = a.narrow(2 - e, G, n[e])
    return a


EVOLVE = dict(gradne_from_state=1, update_te=1, bound_specden=1)  # parameters of a case that takes many steps


def _single(c, seed, **prm):
    mech = mechanism(c["mech"])
    n = (c["nx"], c["ny"], c["nz"])
    te = (0.5, 5.0) if c["mech"] == "argon4" else (0.3, 10.0)
    return Box(mech, _dim(c), n, seed, dens=DENS[c["mech"]], te=te, **prm)


def _boxes(c, seed, serve=False):
    """The uneven boxes of a batch or of a request stream; the sizes are the case's own, the fields the seed's."""
    mech = mechanism(c["mech"])
    sizes = random.Random(f"{c['boxes']} {c['lo']} {c['hi']} {c['steps']}")
    out = []
    for i in range(c["boxes"]):
        ones = c["ones"] if not serve else c["boxes"] // 2  # that many 1-D boxes, the rest 2-D
        dim = 1 if i < ones else 2
        n = [_log(sizes, c["lo"], c["hi"]) if d < dim else 1 for d in range(3)]
        kw = dict(dens=DENS[c["mech"]], precision=PREC[c["precision"]], **EVOLVE)
        if not serve:
            out.append((Box(mech, dim, n, seed * 1000 + i, dt=1e-12, **kw), c["steps"]))
            continue
        # requests differ in voltage, pressure and length; the step is the electrons' drift limit
        v, p = sizes.uniform(500.0, 1500.0), math.exp(sizes.uniform(math.log(0.5), math.log(10.0)))
        steps = _log(sizes, 50, c["steps"]) if c["steps"] > 50 else c["steps"]
        b = Box(mech, dim, n, seed * 1000 + i, voltage=v, bg=2.4e25 * p, dt=1e-13, **kw)
        out.append((b, steps))
    return out


def prepare(c, seed):
    kind = c["kind"]
    if kind == "update":
        kw = dict(EVOLVE) if c["evolve"] else {}
        b = _single(c, seed, blob=c["mech"] == "argon4", dt=1e-12, hyp_order=c["order"], weno_scheme=c["weno"],
                    precision=PREC[c["precision"]], **kw)
        pn, ds, rx = b.dc.new_outputs()
        out = list(pn.unbind(0))
        if c["rates"]:
            out += list(ds.unbind(0)) + list(rx.unbind(0))
        return dict(c=c, b=b, pn=pn, ds=ds if c["rates"] else None, rx=rx if c["rates"] else None, out=out)
    if kind == "percall":
        b = _single(c, seed, blob=c["mech"] == "argon4", dt=1e-12, hyp_order=c["order"], weno_scheme=c["weno"])
        pn, ds, rx = b.dc.new_outputs()
        ns, bg = b.mech.ns, b.mech.bg_species
        return dict(c=c, b=b, pn=pn, rx=rx, flux=[api.face_tensor(b.case, d) for d in range(b.dim)],
                    ds={s: ds[s:s + 1] for s in range(ns + 1) if s not in bg},
                    out=list(rx.unbind(0)) + [ds[s] for s in range(ns + 1) if s not in bg] + [pn[ns + 6], pn[ns + 7]])
    if kind == "coupled":
        b = _single(c, seed, ramp=True, faces=False, dt=1e-12, precision=PREC[c["precision"]], **EVOLVE)
        ns = b.mech.ns
        pn, _, _ = b.dc.new_outputs()
        v = _valid(b.state, b.dim, b.n)
        # potential, field and reduced field of the state, the face fields, and the updated components
        out = [v[ns + 2 + q] for q in range(1 + b.dim)] + [v[ns + 9]] + b.ef[:b.dim] + list(pn.unbind(0))
        return dict(c=c, b=b, pn=pn, pot=b.state[ns + 2].clone(), out=out,
                    pp=api.poisson_params(b.dim, 1000.0, 0.0, max_vcycles=40, tol_rel=1e-10))
    if kind == "species":
        w = c["walls"]
        bc = abi.BC_HNEU if w == "hneu" else abi.BC_IHNEU
        b = _single(c, seed, dt=1e-9 if w == "hneu" else 1e-12, bc=bc, bound_specden=1)
        ns = b.mech.ns
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        old = b.state.clone()
        old[:ns + 1] *= 1.0 + 0.01 * (2 * torch.rand(old[:ns + 1].shape, generator=gen, dtype=torch.float64,
                                                     device="cuda") - 1)
        v = _valid(b.state, b.dim, b.n)[:ns + 1]
        ds = (1e-3 / b.params["dt"]) * v * (2 * torch.rand(v.shape, generator=gen, dtype=torch.float64, device="cuda") - 1)
        spec = {"electron": b.mech.e_id, "ion": 3, "energy": ns}[c["spec"]]
        gn = [api.face_tensor(b.case, d) for d in range(3)] if c["spec"] == "electron" else None
        pn, _, _ = b.dc.new_outputs()
        out = [pn[spec]] + ([pn[ns + 1]] if spec == ns else []) + (gn[:b.dim] if gn else [])
        return dict(c=c, b=b, old=old, ds=ds.contiguous(), pn=pn, spec=spec, gn=gn, out=out)
    if kind == "batch":
        bs = _boxes(c, seed)
        need = sum(api.Batch.case_bytes(b.case, b.prm) for b, _ in bs)
        batch = api.Batch(PREC[c["precision"]], budget_bytes=int(need * 1.02) + (1 << 20), max_cases=len(bs))
        ids = [batch.add(b.hosted(), b.prm, nsteps=n) for b, n in bs]
        outs = [torch.empty_like(b.state) for b, _ in bs]
        return dict(c=c, bs=bs, batch=batch, ids=ids, outs=outs, out=[_parts(o, bs[0][0].mech) for o in outs])
    bs = _boxes(c, seed, serve=True)
    need = sum(api.Batch.case_bytes(b.case, b.prm) for b, _ in bs)
    server = api.Server(PREC[c["precision"]], budget_bytes=int(need * 1.1) + (1 << 20), max_cases=len(bs))
    return dict(c=c, bs=bs, server=server, cases=[(b.hosted(), b.prm, n) for b, n in bs])


def _parts(st, mech):
    """A state as its electrons, background gas, other species, and energy, temperature and fields."""
    return [st[0], st[1], st[2:mech.ns], st[mech.ns], st[mech.ns + 1], st[mech.ns + 2:mech.ns + 6], st[mech.ns + 6:]]


# ---------------------------------------------------------------------------
# one pass


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "update":
        api.explicit_update_all(s["b"].dc, s["b"].prm, s["pn"], s["ds"], s["rx"])
        return s["out"]
    if kind == "percall":
        b = s["b"]
        api.reaction_source(b.dc, s["rx"])
        for sp, ds in s["ds"].items():
            for d in range(b.dim):
                api.compute_explicit_flux(b.dc, d, sp, s["flux"][d], hyp_order=c["order"], weno=c["weno"])
            api.compute_dsdt(b.dc, sp, s["flux"], s["rx"], ds)
        api.compute_elecenergy_source(b.dc, s["rx"], s["ds"][b.mech.ns], s["pn"], b.prm)
        return s["out"]
    if kind == "coupled":
        b = s["b"]
        b.state[b.mech.ns + 2].copy_(s["pot"])  # the initial guess: the potential the step began with
        api.poisson_solve(b.dc, b.prm, s["pp"])
        scales = api.time_scales(b.dc, b.prm)
        api.explicit_update_all(b.dc, b.prm, s["pn"])
        return s["out"] + [*scales]
    if kind == "species":
        api.implicit_species_solve(s["b"].dc, s["spec"], s["old"], s["ds"], s["pn"], s["b"].prm, gradne=s["gn"],
                                   tol_rel=1e-10)
        return s["out"]
    if kind == "batch":
        batch = s["batch"]
        for cid, (b, n) in zip(s["ids"], s["bs"]):
            batch.load(cid, b.state, nsteps=n)
        batch.step(c["steps"])
        for cid, o in zip(s["ids"], s["outs"]):
            batch.read(cid, out=o)
        return [x for o in s["out"] for x in (o if len(s["out"]) <= 9 else _merge(o))]
    srv = s["server"]
    rids = [srv.submit(case, prm, n) for case, prm, n in s["cases"]]
    return [x for r in rids for x in _parts(srv.wait(r)[0], s["bs"][0][0].mech)]


def _merge(o):
    """At most four outputs per box, so that 16 boxes stay within 64."""
    return [o[0], o[2], o[3], o[4]]


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _update_work(dim, ns, nr, cells, nflux, order, rates=0):
    per = 8.0 * (ns + 2 + dim + 2 * dim + ns + 1 + (2 * (ns + 1) if rates else 0))
    weno = {5: 2 * 95, 2: 20, 1: 10}[order]
    return per * cells, float(cells) * (nflux * dim * weno + nr * 25 + 3 * ns)


def work(c):
    ns, nr = MECHS[c["mech"]]
    nflux = 3 if c["mech"] == "argon4" else 2 + (ns - 2) // 2  # electrons, ions, electron energy
    if c["kind"] in ("batch", "serve"):
        sizes = random.Random(f"{c['boxes']} {c['lo']} {c['hi']} {c['steps']}")
        by = fl = 0.0
        for i in range(c["boxes"]):
            dim = 1 if i < (c["ones"] if c["kind"] == "batch" else c["boxes"] // 2) else 2
            n = [_log(sizes, c["lo"], c["hi"]) for _ in range(dim)]
            steps = c["steps"]
            if c["kind"] == "serve":
                sizes.uniform(500.0, 1500.0), sizes.uniform(0.0, 1.0)
                steps = _log(sizes, 50, c["steps"]) if c["steps"] > 50 else c["steps"]
            x, y = _update_work(dim, ns, nr, math.prod(n), nflux, 5)
            by, fl = by + steps * x, fl + steps * y
        return {"bytes": by, "flops": fl}
    dim, cells = _dim(c), c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "species":  # state in, old, dsdt, solution and Te out; two smoothing cycles at least
        return {"bytes": 8.0 * cells * (ns + 6 + dim), "flops": cells * 200.0}
    by, fl = _update_work(dim, ns, nr, cells, nflux, c.get("order", 5), c.get("rates", 0))
    if c["kind"] == "percall":  # each flux is written and read, dsdt written
        by += 8.0 * cells * ((ns - 1 + 1) * (2 * dim + 1))
    if c["kind"] == "coupled":  # charge density in; potential, field, reduced field and face fields out
        by += 8.0 * cells * (ns + 3 + 2 * dim)
        fl += cells * 300.0
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch

N_A, NA_CE = 6.02214076e23, 6.02214085774e23
K_B, PI, ECHARGE, ME = 1.380649e-23, math.pi, 1.60217662e-19, 9.10938188e-31
M_AMU, EPS0, EV2J = 1.66054e-27, 8.854187817e-12, 1.602176620800000e-19
EV = ECHARGE / K_B


def _mob(m, s, te, nd, tg):
    k = m.mob_kind[s]
    if k == abi.MOB_SCALED:
        return m.mob_p0[s] * _mob(m, m.mob_ref[s], te, nd, tg)
    if k == abi.MOB_ELECTRON:
        return (-ECHARGE / ME) / math.sqrt(8 * K_B / PI / ME) / (torch.sqrt(te) * nd * m.mob_p0[s])
    if k == abi.MOB_ION_TG:
        w = m.mob_p1[s]
        return (ECHARGE / w) / math.sqrt(8 * K_B / PI / w) / (math.sqrt(tg) * nd * m.mob_p0[s])
    return None  # no drift


def _diff(m, s, te, nd, tg):
    mu = _mob(m, m.diff_ref[s], te, nd, tg)
    if m.diff_kind[s] == abi.DIFF_TE_ABSMOB:
        return m.diff_factor[s] * (te / EV) * mu.abs()
    return m.diff_factor[s] * (tg / EV) * mu


def _chemistry(m, v, tg):
    """rxn (NS+1) of the valid cells."""
    ns = m.ns
    te = v[ns + 1]
    sc = v[:ns] / N_A
    w = torch.zeros_like(v[:ns + 1])
    mee = 1.5 * te * K_B * NA_CE
    sefact = (torch.tanh((te - tg) / 0.5) + 1.0) / 2.0
    dt = te - tg
    for r in m.reactions:
        k = torch.exp(math.log(r.A) + r.b * torch.log(te) - r.C / te)
        q = k
        for s in r.reactants:
            q = q * sc[s]
        for s, coef in r.terms:
            w[s] += coef * q
        if r.rxntype in (abi.RXN_EXCITATION, abi.RXN_IONIZATION):
            w[ns] -= (r.eexci * EV2J) * NA_CE * q * sefact
        elif r.rxntype == abi.RXN_RECOMB:
            w[ns] -= mee * q
        elif r.rxntype == abi.RXN_ELASTIC:
            w[ns] -= 3.0 * K_B * (m.mw[m.e_id] / m.mw[r.elidx]) * dt * (sc[m.e_id] * sc[r.elidx] * k) * NA_CE
    nu = -ECHARGE / ME / _mob(m, m.e_id, te, v[:ns].sum(0), tg)
    w[ns] -= 1.5 * K_B * v[m.e_id] * dt * nu * (2.0 * ME / m.elastic_mass)
    w[:ns] *= N_A
    return w


def _weno(a, b, c, d, e, scheme):
    eps = 1e-20
    p = (a / 3 - 7 / 6 * b + 11 / 6 * c, -b / 6 + 5 / 6 * c + d / 3, c / 3 + 5 / 6 * d - e / 6)
    be = (13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
          13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
          13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2)
    g = (0.1, 0.6, 0.3)
    if scheme == 3:
        tau = (be[0] - be[2]).abs()
        al = [g[k] * (1 + (tau / (be[k] + eps)) ** 2) for k in range(3)]
    else:
        al = [g[k] / (be[k] + eps) ** 2 for k in range(3)]
        if scheme == 2:
            t = al[0] + al[1] + al[2]
            al = [w * (q + q * q - 3 * q * w + w * w) / (q * q + w * (1 - 2 * q)) for w, q in zip((x / t for x in al), g)]
    t = al[0] + al[1] + al[2]
    return sum(x / t * y for x, y in zip(al, p))


def _face_flux(u, v, order, scheme, dt):
    """Flux from the stencil values u, v: six tensors each, cells f-3 .. f+2."""
    if order == 1:
        sg = torch.sign(0.5 * (v[2] + v[3]))
        sg = torch.where(sg == 0, torch.ones_like(sg), sg)
        return u[2] * v[2] * 0.5 * (1 + sg) + u[3] * v[3] * 0.5 * (1 - sg)
    if order == 2:
        dl, dm, dr = u[2] - u[1], u[3] - u[2], u[4] - u[3]
        vm = 0.5 * (v[2] + v[3])
        sg = torch.where(vm >= 0, 1.0, -1.0)
        cfl = vm * dt / DX
        r = torch.where(cfl >= 0, dl, dr) / (dm + 1e-30)
        lim = torch.where(r <= 0, torch.ones_like(r), torch.where(r <= 1, 1 - (1 - cfl.abs()) * r, cfl.abs()))
        fl, fr = u[2] * v[2], u[3] * v[3]
        return 0.5 * (fl + fr) - 0.5 * sg * lim * (fr - fl)
    f = [x * y for x, y in zip(u, v)]
    lam = (0.5 * (v[2] + v[3])).abs()
    return 0.5 * (_weno(*f[:5], scheme) + lam * _weno(*u[:5], scheme)) + 0.5 * (
        _weno(*f[:0:-1], scheme) - lam * _weno(*u[:0:-1], scheme))


def _step(b, st, ef, gn, order, weno, dsdt_only=False):
    """(updated valid components, dsdt, rxn) of one explicit step from the ghosted state st."""
    m, dim, n, prm = b.mech, b.dim, b.n, b.prm
    ns, tg, dt = m.ns, prm.Tg, prm.dt
    v = _valid(st, dim, n)
    rxn = _chemistry(m, v, tg)
    ds = rxn.clone()
    nd, te = st[:ns].sum(0), st[ns + 1]
    for s in range(ns + 1):
        mu = None if s in m.bg_species else _mob(m, s, te, nd, tg)
        if mu is None:
            continue
        for d in range(dim):
            ax = 2 - d
            u, w = _valid_but(st[s], dim, n, d), _valid_but(mu * st[ns + 3 + d], dim, n, d)
            F = _face_flux([u.narrow(ax, q, n[d] + 1) for q in range(6)], [w.narrow(ax, q, n[d] + 1) for q in range(6)],
                           order, weno, dt)
            F.narrow(ax, 0, 1).zero_()  # walls without a drift flux
            F.narrow(ax, n[d], 1).zero_()
            ds[s] += (F.narrow(ax, 0, n[d]) - F.narrow(ax, 1, n[d])) / DX
    # Joule heating: half the sum over the cell's faces, a domain face replaced by the next one inward
    jh = torch.zeros_like(v[0])
    for d in range(dim):
        ax = 2 - d

        def avg(x):
            p = _valid_but(x, dim, n, d)
            return 0.5 * (p.narrow(ax, G - 1, n[d] + 1) + p.narrow(ax, G, n[d] + 1))

        tf, nf = avg(te), avg(nd)
        ne = _valid_but(st[m.e_id], dim, n, d)
        g = (ne.narrow(ax, G, n[d] + 1) - ne.narrow(ax, G - 1, n[d] + 1)) / DX if prm.gradne_from_state else gn[d][0]
        e = ef[d][0]
        J = -ECHARGE * (_mob(m, m.e_id, tf, nf, tg) * avg(st[m.e_id]) * e - _diff(m, m.e_id, tf, nf, tg) * g) * e
        J.narrow(ax, 0, 1).copy_(J.narrow(ax, 1, 1))
        J.narrow(ax, n[d], 1).copy_(J.narrow(ax, n[d] - 1, 1))
        jh += J.narrow(ax, 0, n[d]) + J.narrow(ax, 1, n[d])
    jh *= 0.5
    ds[ns] += jh
    pn = v.clone()
    for s in range(ns + 1):
        if s in m.bg_species:
            continue
        pn[s] = v[s] + dt * ds[s]
        if prm.bound_specden and s != ns:
            pn[s].clamp_(min=1e10)
    if prm.update_te:
        t = (2.0 / 3.0) / K_B * pn[ns] / v[m.e_id]
        cold = t < 300.0
        t = torch.where(cold, torch.full_like(t, 300.0), t)
        pn[ns] = torch.where(cold, 1.5 * K_B * pn[m.e_id] * t, pn[ns])
        pn[ns + 1] = t
    pn[ns + 6], pn[ns + 7] = jh, rxn[ns]
    return pn, ds, rxn


def _advance(b, steps):
    """The ghosted state after some steps, its ghosts refilled after each."""
    st, ns = b.state.clone(), b.mech.ns
    for _ in range(steps):
        pn, _, _ = _step(b, st, b.ef, b.gn, 5, 3)
        _valid(st, b.dim, b.n).copy_(pn)
        for s in list(range(ns)) + [ns, ns + 1]:
            for d in range(b.dim):
                p = _valid_but(st[s], b.dim, b.n, d)
                ax = 2 - d
                for q in range(1, G + 1):
                    p.narrow(ax, G - q, 1).copy_(p.narrow(ax, G, 1))
                    p.narrow(ax, G + b.n[d] - 1 + q, 1).copy_(p.narrow(ax, G + b.n[d] - 1, 1))
    return st


def _lap(phi, dim, n):
    """(sum of the neighbours' differences)/dx^2 with a fixed potential (1000 V, 0 V) at the x faces."""
    out = torch.zeros_like(phi)
    for d in range(dim):
        ax = 2 - d
        g = (phi.narrow(ax, 1, n[d] - 1) - phi.narrow(ax, 0, n[d] - 1)) / DX
        out.narrow(ax, 0, n[d] - 1).add_(g / DX)
        out.narrow(ax, 1, n[d] - 1).sub_(g / DX)
    out[..., 0] += 2 * (1000.0 - phi[..., 0]) / DX**2
    out[..., -1] += 2 * (0.0 - phi[..., -1]) / DX**2
    return out


def _potential(b):
    """The discrete potential by its eigenvectors (sines along x, cosines across), refined twice."""
    m, dim, n = b.mech, b.dim, b.n
    v = _valid(b.state, dim, n)
    rhs = torch.zeros_like(v[0])
    for s in range(m.ns):
        if m.charge[s]:
            rhs += m.charge[s] * v[s]
    rhs *= -ECHARGE / EPS0
    Q, lam = [], []
    for d in range(dim):
        i = torch.arange(n[d], device="cuda", dtype=torch.float64)
        k = i + 1 if d == 0 else i
        ang = PI * k[:, None] * (i[None, :] + 0.5) / n[d]
        q = torch.sin(ang) if d == 0 else torch.cos(ang)
        Q.append(q / q.norm(dim=1, keepdim=True))
        lam.append(-4.0 / DX**2 * torch.sin(PI * k / (2 * n[d])) ** 2)
    tot = sum(x.reshape([-1 if e == 2 - d else 1 for e in range(3)]) for d, x in enumerate(lam))

    def apply(x, inv):
        for d in range(dim):
            x = torch.tensordot(x, Q[d].t() if not inv else Q[d], dims=([2 - d], [0])).movedim(-1, 2 - d)
        return x

    phi = torch.zeros_like(rhs)
    for _ in range(3):
        phi = phi + apply(apply(rhs - _lap(phi, dim, n), False) / tot, True)
    return phi


def _coupled(c, b):
    m, dim, n = b.mech, b.dim, b.n
    ns = m.ns
    phi = _potential(b)
    v = _valid(b.state, dim, n)
    v[ns + 2] = phi
    e2 = 0.0
    ef = []
    for d in range(dim):
        ax, N = 2 - d, n[d]
        P = lambda i: phi.narrow(ax, i, 1)  # noqa: E731
        e = torch.empty_like(phi)
        e.narrow(ax, 1, N - 2).copy_(-0.5 * (phi.narrow(ax, 2, N - 2) - phi.narrow(ax, 0, N - 2)) / DX)
        e.narrow(ax, 0, 1).copy_(-0.5 * (-P(2) + 4 * P(1) - 3 * P(0)) / DX)
        e.narrow(ax, N - 1, 1).copy_(-0.5 * (P(N - 3) - 4 * P(N - 2) + 3 * P(N - 1)) / DX)
        v[ns + 3 + d] = e
        e2 = e2 + e * e
        f = torch.zeros(b.ef[d].shape[1:], dtype=torch.float64, device="cuda")
        f.narrow(ax, 1, N - 1).copy_(-(phi.narrow(ax, 1, N - 1) - phi.narrow(ax, 0, N - 1)) / DX)
        if d == 0:
            f.narrow(ax, 0, 1).copy_(-(P(0) - 1000.0) / (0.5 * DX))
            f.narrow(ax, N, 1).copy_(-(0.0 - P(N - 1)) / (0.5 * DX))
        ef.append(f[None])
    v[ns + 9] = torch.sqrt(e2) / v[:ns].sum(0) / 1e-21
    out = [v[ns + 2 + q].clone() for q in range(1 + dim)] + [v[ns + 9].clone()] + ef
    te, nd, tg = v[ns + 1], v[:ns].sum(0), b.prm.Tg
    mu, dc, em = _mob(m, m.e_id, te, nd, tg).abs(), _diff(m, m.e_id, te, nd, tg), torch.sqrt(e2)
    scales = [DX / float((mu * em).max()), 0.5 * DX * DX / float(dc.max()) / dim,
              EPS0 / ECHARGE / float((mu * v[m.e_id]).max())]
    before = v.clone()
    before[ns + 2], before[ns + 3:] = 0.0, 0.0
    _ghosts(b.state, dim, n)
    pn, _, _ = _step(b, b.state, ef + b.ef[dim:], b.gn, 5, 3)
    # the fields belong to the state: the update leaves the output's own as they were
    ramp = 1000.0 * (1.0 - (torch.arange(n[0], device="cuda", dtype=torch.float64) + 0.5) / n[0])
    pn[ns + 2] = ramp[None, None, :]
    for q in (3, 4, 5, 8, 9):
        pn[ns + q] = 0.0
    return out + list(pn.unbind(0)) + scales


def _species(c, s):
    """The implicit solve by conjugate gradients."""
    b, spec = s["b"], s["spec"]
    m, dim, n, prm = b.mech, b.dim, b.n, b.prm
    ns, tg, dt = m.ns, prm.Tg, prm.dt
    st = b.state
    D = _diff(m, spec, st[ns + 1], st[:ns].sum(0), tg)
    x = _valid(st, dim, n)
    rhs = _valid(s["old"], dim, n)[spec] / dt + s["ds"][spec]
    B, wall = [], []
    for d in range(dim):
        ax = 2 - d
        p = _valid_but(D, dim, n, d)
        l, r = p.narrow(ax, G - 1, n[d] + 1), p.narrow(ax, G, n[d] + 1)
        f = 2 * l * r / (l + r)
        B.append(f)
        g = [None, None]
        if c["walls"] == "ihneu":
            for side, i, sg in ((0, 0, -1.0), (1, n[d] - 1, 1.0)):
                at = lambda a: a.narrow(ax, i, 1)  # noqa: E731
                te, dl = at(x[ns + 1]), at(_valid(D, dim, n))
                cbar = torch.sqrt(8 * K_B * te / PI / ME)
                if spec == m.e_id:
                    g[side] = -(at(x[m.e_id]) * cbar / 4 * sg) / dl
                elif spec == ns:
                    g[side] = -(2 * K_B * te * at(x[m.e_id]) * cbar / 4 * sg) / dl
                else:
                    drift = _mob(m, spec, te, at(x[:ns].sum(0)), tg) * at(x[spec]) * at(x[ns + 3 + d])
                    g[side] = torch.where(drift * sg >= 0, -drift / dl, torch.zeros_like(drift))
                rhs.narrow(ax, i, 1).add_(sg * f.narrow(ax, 0 if side == 0 else n[d], 1) * g[side] / DX)
        wall.append(g)

    def A(y):
        out = y / dt
        for d in range(dim):
            ax = 2 - d
            q = B[d].narrow(ax, 1, n[d] - 1) * (y.narrow(ax, 1, n[d] - 1) - y.narrow(ax, 0, n[d] - 1)) / DX**2
            out.narrow(ax, 0, n[d] - 1).sub_(q)
            out.narrow(ax, 1, n[d] - 1).add_(q)
        return out

    y = x[spec].clone()
    for _ in range(3):  # restarted: the residual is formed anew
        r = rhs - A(y)
        p, rr = r.clone(), (r * r).sum()
        e = torch.zeros_like(y)
        for it in range(400):
            q = A(p)
            al = rr / (p * q).sum()
            e += al * p
            r -= al * q
            new = (r * r).sum()
            if it % 20 == 19 and float(new) <= 1e-26 * float((rhs * rhs).sum()):
                break
            p = r + (new / rr) * p
            rr = new
        y = y + e
    if spec != ns:
        y.clamp_(min=1e10)
    out = [y]
    if spec == ns:
        t = (2.0 / 3.0) / K_B * y / x[m.e_id]
        t0 = t.clamp(min=300.0)
        out = [torch.where(t < 300.0, 1.5 * K_B * x[m.e_id] * t0, y), t0]
    if spec == m.e_id:
        for d in range(dim):
            ax = 2 - d
            g = torch.zeros(s["gn"][d].shape[1:], dtype=torch.float64, device="cuda")
            g.narrow(ax, 1, n[d] - 1).copy_((y.narrow(ax, 1, n[d] - 1) - y.narrow(ax, 0, n[d] - 1)) / DX)
            if wall[d][0] is not None:
                g.narrow(ax, 0, 1).copy_(wall[d][0])
                g.narrow(ax, n[d], 1).copy_(wall[d][1])
            out.append(g[None])
    return out


def exact(c, seed):
    kind = c["kind"]
    if kind in ("batch", "serve"):
        bs = _boxes(c, seed, serve=kind == "serve")
        if sum(b.n[0] * b.n[1] * n for b, n in bs) > 4e8 or sum(n for _, n in bs) > 700:
            return None
        parts = [_parts(_advance(b, n), b.mech) for b, n in bs]
        if kind == "batch" and len(parts) > 9:
            parts = [_merge(p) for p in parts]
        return [x for p in parts for x in p]
    s = prepare(c, seed)
    b = s["b"]
    if kind == "coupled":
        return _coupled(c, b)
    if kind == "species":
        return _species(c, s)
    pn, ds, rxn = _step(b, b.state, b.ef, b.gn, c["order"], c["weno"])
    if kind == "update":
        return list(pn.unbind(0)) + (list(ds.unbind(0)) + list(rxn.unbind(0)) if c["rates"] else [])
    ns, bg = b.mech.ns, b.mech.bg_species
    return list(rxn.unbind(0)) + [ds[q] for q in range(ns + 1) if q not in bg] + [pn[ns + 6], pn[ns + 7]]
