"""The work that users of this framework have it do, as cases that can be timed and compared.

Kinds of case, each through the entry points that a driver program calls:

  steps      ``Context.rk3_steps``: RK3 steps with in-kernel noise, replayed from the context's graph
  full       ``Context.rk3_step(aux=True)``: the reference's RK3stepStag call with all its by-products
  operators  conservedToPrimitiveStag, FillBoundary, calculateTransportCoeffs, calculateFluxStag one by one
  ensemble   ``Batch.step``: many independent runs advanced together
  stats      ``Context.stats_stag``: the running statistics after a step, with the x-line correlations
  structfact ``StructFact``: samples of the structure factor and its output

``exact`` restates each kind in plain torch in 64 bits.
"""
import math
import random

import torch

from fhdex_b200 import capi
from fhdex_b200.batch import Batch
from fhdex_b200.context import Context
from fhdex_b200.fab import CELL, EDGE, FACE, MultiFab
from fhdex_b200.params import argon, argon_single, mixture4, no2_dimerization, stable_dt, with_walls
from fhdex_b200.state import StagState
from fhdex_b200.stats import StatsState
from fhdex_b200.structfact import StructFact

GASES = {"argon": argon, "single": argon_single, "mixture4": mixture4, "no2": no2_dimerization}


def _case(name, kind, gas, n, **kw):
    return dict(name=name, kind=kind, gas=gas, nx=n[0], ny=n[1], nz=n[2], **kw)


def listed():
    return [
        # the smallest boxes that runs are served at: launches and latency
        _case("step_argon16", "steps", "argon", (16, 16, 16), mixed=False, walls="none", steps=10),
        # the plain method's box, 32^3 in FP64
        _case("step_argon32", "steps", "argon", (32, 32, 32), mixed=False, walls="none", steps=10),
        # a served one-species request with a ragged box, mixed precision
        _case("step_single61_mixed", "steps", "single", (61, 47, 53), mixed=True, walls="none", steps=5),
        # the large-grid method, FP64
        _case("step_argon128", "steps", "argon", (128, 128, 128), mixed=False, walls="none", steps=2),
        # the headline box, FP64
        _case("step_argon256", "steps", "argon", (256, 256, 256), mixed=False, walls="none", steps=1),
        # the 4-species mixture in mixed precision
        _case("step_mix128_mixed", "steps", "mixture4", (128, 128, 128), mixed=True, walls="none", steps=2),
        # a temperature gradient between no-slip isothermal x walls, as the regression decks have it
        _case("step_walls96", "steps", "argon", (96, 64, 64), mixed=False, walls="noslip", steps=2),
        # the drop-in call of a driver that plots fluxes and coefficients, with reactions
        _case("full_no2_100", "full", "no2", (100, 84, 75), mixed=False),
        # the operators that a driver of its own time stepper calls, four species in FP64
        _case("operators_mix72", "operators", "mixture4", (72, 65, 54), mixed=False),
        # an ensemble, half 32^3 and half 64^3, each member with its own gas state
        _case("ensemble48_mixed", "ensemble", "argon", (32, 32, 32), mixed=True, members=48, steps=1),
        # the running statistics of a 3-D run with plot_cross
        _case("stats_argon144", "stats", "argon", (144, 112, 96), cross=True),
        # the structure factor of four variables: samples and the output
        _case("structfact144", "structfact", "argon", (144, 112, 96), samples=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["full", "operators", "ensemble", "stats", "structfact"])
    if kind == "steps":
        gas = rng.choice(["argon", "argon", "single", "mixture4", "no2"])
        walls = rng.choice(["none", "none", "none", "noslip", "slip"]) if gas in ("argon", "mixture4") else "none"
        # four species in FP64 cost several times as much per cell
        e = _log(rng, 16, 88 if gas == "mixture4" else 136)
        n = [max(12, int(e * rng.uniform(0.75, 1.25))) for _ in range(3)]
        steps = max(1, min(10, int(4e6 / (n[0] * n[1] * n[2]))))
        return dict(kind=kind, gas=gas, nx=n[0], ny=n[1], nz=n[2], mixed=walls == "none" and rng.random() < 0.4,
                    walls=walls, steps=steps)
    if kind == "ensemble":
        e = rng.randint(16, 36)
        return dict(kind=kind, gas=rng.choice(["argon", "argon", "single"]), nx=e, ny=e, nz=e,
                    mixed=rng.random() < 0.7, members=rng.randint(8, 40), steps=rng.randint(1, 2))
    e = _log(rng, 24, 112)
    n = [max(12, int(e * rng.uniform(0.75, 1.25))) for _ in range(3)]
    c = dict(kind=kind, gas=rng.choice(["argon", "mixture4"] if kind != "full" else ["argon", "no2", "mixture4"]),
             nx=n[0], ny=n[1], nz=n[2])
    if kind in ("full", "operators"):
        c["mixed"] = False
    if kind == "stats":
        c["cross"] = rng.random() < 0.5
    if kind == "structfact":
        c["samples"] = rng.randint(1, 3)
    return c


# ---- inputs ------------------------------------------------------------------------------


def _device():
    return "cuda:0" if torch.cuda.is_available() else "cpu"


def _params(case, seed, n=None, **kw):
    n = n or (case["nx"], case["ny"], case["nz"])
    dx = 1e-5 if case["gas"] == "no2" else 8e-6
    p = GASES[case["gas"]](n, dx=dx, precision=int(bool(case.get("mixed"))), seed=seed, **kw)
    walls = case.get("walls", "none")
    if walls == "noslip":
        p = with_walls(p, x=dict(vel=2, therm=2, mass=1, t=(0.9 * p.T_init, 1.1 * p.T_init)))
    elif walls == "slip":
        p = with_walls(p, x=dict(vel=1, therm=1, mass=1))
    return p


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _wall_x(p):
    return bool(p.walls) and p.bc_vel_lo[0] != -1


def _wrap(p, a, nodal):
    """The duplicate points n of the nodal periodic directions take the value of the points 0."""
    for d in range(3):
        if nodal[d] and not (d == 0 and _wall_x(p)):
            a.select(-1 - d, p.n_cells[d]).copy_(a.select(-1 - d, 0))
    return a


def _normal(p, g, nodal=CELL, lead=()):
    shape = tuple(lead) + tuple(p.n_cells[d] + nodal[d] for d in (2, 1, 0))
    return _wrap(p, torch.randn(shape, generator=g, device=_device(), dtype=torch.float64), nodal)


def _fluctuations(p, g):
    """A state with the equilibrium's own fluctuations: valid densities, temperature and face momenta."""
    dv = p.dx[0] * p.dx[1] * p.dx[2]
    rho_k = []
    for k in range(p.nspecies):
        mean = p.rho0 * p.rhobar[k]
        number = mean / (p.molmass[k] * p.k_B / p.Runiv) * dv
        rho_k.append(mean * (1.0 + _normal(p, g) / math.sqrt(number)))
    hcv, _ = p.hc()
    cv = sum(p.rhobar[k] * hcv[k] for k in range(p.nspecies))
    temp = p.T_init * (1.0 + math.sqrt(p.k_B / (p.rho0 * cv * dv)) * _normal(p, g))
    mom = [math.sqrt(p.rho0 * p.k_B * p.T_init / dv) * _normal(p, g, FACE[d]) for d in range(3)]
    if _wall_x(p):
        mom[0][..., 0] = 0.0
        mom[0][..., -1] = 0.0
    return rho_k, temp, mom


def _conserved(p, rho_k, temp, mom):
    """(rho, rhoE) of the valid cells."""
    hcv, _ = p.hc()
    rho = sum(rho_k)
    energy = sum(r * (p.e0[k] + hcv[k] * temp) for k, r in enumerate(rho_k))
    kin = sum((_lo(m, d) + _hi(m, d)) ** 2 for d, m in enumerate(mom))
    return rho, energy + 0.125 * kin / rho


def _lo(a, d):
    return a.narrow(-1 - d, 0, a.shape[-1 - d] - 1)


def _hi(a, d):
    return a.narrow(-1 - d, 1, a.shape[-1 - d] - 1)


def _load(ctx, st, p, fluct):
    """main_driver's initialisation with the given valid state."""
    rho_k, temp, mom = fluct
    ctx.init_cons_var_stag(st)
    rho, energy = _conserved(p, rho_k, temp, mom)
    st.cu.valid(0).copy_(rho)
    st.cu.valid(4).copy_(energy)
    for k, r in enumerate(rho_k):
        st.cu.valid(5 + k).copy_(r)
    for d in range(3):
        st.cumom[d].valid(0).copy_(mom[d])
    for m in [st.cu] + st.cumom:
        ctx.fill_boundary(m)
    ctx.conserved_to_primitive(st)
    for m in [st.cu, st.prim] + st.cumom + st.vel:
        ctx.fill_boundary(m)
    if p.walls:
        ctx.set_bc(st)


def _member_params(case, seed):
    """The members of an ensemble: half at the case's edge, half at twice that."""
    rng = random.Random(seed)
    out = []
    for q in range(case["members"]):
        e = case["nx"] if q < case["members"] // 2 else 2 * case["nx"]
        out.append(_params(case, (seed << 20) + q + 1, n=(e, e, e), T_init=rng.uniform(250.0, 350.0),
                           rho0=rng.uniform(1e-3, 3e-3)))
    return out


def _operator_noise(p, g):
    """W of one flux evaluation: faces (energy, species), edges and centres."""
    return ([_normal(p, g, FACE[d], (p.nspecies + 1,)) for d in range(3)], [_normal(p, g, EDGE[e]) for e in range(3)],
            [math.sqrt(2.0) * _normal(p, g) for d in range(3)])


SF_NAMES = ["rho", "rhoE", "T", "jx"]
SF_PAIRS = len(SF_NAMES) * (len(SF_NAMES) + 1) // 2


def _sf_variables(p, g):
    rho_k, temp, mom = _fluctuations(p, g)
    rho, energy = _conserved(p, rho_k, temp, mom)
    return torch.stack([rho, energy, temp, _lo(mom[0], 0)])


def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    dev = _device()
    if kind == "ensemble":
        params = _member_params(case, seed)
        batch = Batch(params[0].nspecies, int(bool(case["mixed"])), 0)
        # the members' MultiFabs lie in one tensor per field, as an ensemble's program keeps them
        fields = {"cu": [], "mom": [], "prim": [], "vel": []}
        states = [StagState(p, "meta", aux=False) for p in params]
        for st in states:
            for key, mfs in zip(fields, ([st.cu], st.cumom, [st.prim], st.vel)):
                fields[key] += mfs
        flat = {}
        for key, mfs in fields.items():
            flat[key] = torch.zeros(sum(m.arr.numel() for m in mfs), dtype=torch.float64, device=dev)
            at = 0
            for m in mfs:
                size = m.arr.numel()
                m.arr = flat[key][at:at + size].view(m.arr.shape)
                at += size
        for p, st in zip(params, states):
            ctx = Context(p, 0)
            _load(ctx, st, p, _fluctuations(p, g))
            batch.add(p, st, stable_dt(p), init=False)
            ctx.close()
        return {"kind": kind, "batch": batch, "flat": flat, "steps": case["steps"]}
    p = _params(case, seed)
    if kind == "structfact":
        var = []
        for _ in range(case["samples"]):
            m = MultiFab(p.n_cells, CELL, len(SF_NAMES), 0, device=dev)
            m.arr.copy_(_sf_variables(p, g))
            var.append(m)
        return {"kind": kind, "sf": StructFact(p.n_cells, SF_NAMES, [1.0] * SF_PAIRS), "variables": var}
    ctx = Context(p, 0)
    st = StagState(p, dev, aux=kind in ("full", "operators"))
    _load(ctx, st, p, _fluctuations(p, g))
    s = {"kind": kind, "ctx": ctx, "st": st, "dt": stable_dt(p), "step": 0}
    if kind == "steps":
        s["steps"] = case["steps"]
    elif kind == "operators":
        s["noise"] = []
        for lattice, ws in zip((FACE, EDGE, (CELL,) * 3), _operator_noise(p, g)):
            mfs = []
            for nodal, w in zip(lattice, ws):
                m = MultiFab(p.n_cells, nodal, w.shape[0] if w.dim() == 4 else 1, 1 if nodal == CELL else 0, device=dev)
                m.valid().copy_(w)
                ctx.fill_boundary(m)
                mfs.append(m)
            s["noise"].append(mfs)
    elif kind == "stats":
        stats = StatsState(p, dev, cross=case["cross"])
        s["flags"] = 15 | (capi.STATS_CROSS if case["cross"] else 0)
        s["stats"] = stats
        ctx.stats_stag(st, stats, 1, s["flags"])
        _load(ctx, st, p, _fluctuations(p, g))
        s["step"] = 1
    return s


def _state_outputs(st):
    return {"cu": st.cu.arr, "mom": [m.arr for m in st.cumom], "prim": st.prim.arr, "vel": [m.arr for m in st.vel]}


def run(s):
    kind = s["kind"]
    if kind == "steps":
        s["ctx"].rk3_steps(s["st"], s["dt"], s["step"], s["steps"])
        s["step"] += s["steps"]
        return _state_outputs(s["st"])
    if kind == "full":
        st = s["st"]
        s["ctx"].rk3_step(st, s["dt"], s["step"], aux=True)
        s["step"] += 1
        out = _state_outputs(st)
        out.update(coef=[m.arr for m in (st.eta, st.zeta, st.kappa, st.chi, st.D)], source=st.source.arr,
                   faceflux=[m.arr for m in st.faceflux], edgeflux=[m.arr for m in st.edgeflux],
                   cenflux=[m.arr for m in st.cenflux])
        return out
    if kind == "operators":
        ctx, st = s["ctx"], s["st"]
        ctx.conserved_to_primitive(st)
        for m in [st.cu, st.prim] + st.vel:
            ctx.fill_boundary(m)
        ctx.transport_coeffs(st)
        ctx.flux_stag(st, *s["noise"], s["dt"])
        return {"prim": st.prim.arr, "vel": [m.arr for m in st.vel],
                "coef": [m.arr for m in (st.eta, st.zeta, st.kappa, st.chi, st.D)],
                "faceflux": [m.arr for m in st.faceflux], "edgeflux": [m.arr for m in st.edgeflux],
                "cenflux": [m.arr for m in st.cenflux]}
    if kind == "ensemble":
        s["batch"].step(s["steps"])
        s["batch"].synchronize()
        return s["flat"]
    if kind == "stats":
        s["step"] += 1
        stats = s["stats"]
        s["ctx"].stats_stag(s["st"], stats, s["step"], s["flags"])
        out = {k: m.arr for k, m in stats.named().items()}
        if stats.spatialCross is not None:
            out["spatialCross"] = stats.spatialCross
            out["dataSliceMeans_xcross"] = stats.dataSliceMeans_xcross
        return out
    for var in s["variables"]:
        s["sf"].fort_structure(var)
    return [m.arr for m in s["sf"].finalize()]


# ---- what a pass cannot do without --------------------------------------------------------


def _step_flops(p):
    """FP operations of one cell and RK3 step: the transport solves, six faces' worth of fluxes (three
    directions), nine stresses and the combination, each counted from the formulas, three stages."""
    ns = p.nspecies
    transport = 60 + 40 * ns + 45 * ns * ns + 12 * ns ** 3
    faces = 3 * (90 + 45 * ns + 22 * ns * ns)
    return 3 * (transport + faces + 220 + 20 * (5 + ns))


def work(case):
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "ensemble":
        half = case["members"] // 2
        cells *= half + 8 * (case["members"] - half)
    p = _params(case, 1)
    ns, nv, npv = p.nspecies, p.nvars, p.nprimvars
    state_in, state_out = 5 + ns, nv + npv + 6
    coef = 3 + ns + ns * ns
    if kind in ("steps", "ensemble"):
        return {"bytes": 8 * cells * case["steps"] * (state_in + state_out), "flops": cells * case["steps"] * _step_flops(p)}
    if kind == "full":
        flux = 3 * (nv + 4) + 6 + 3
        return {"bytes": 8 * cells * (state_in + state_out + coef + flux + ns), "flops": cells * _step_flops(p)}
    if kind == "operators":
        flux = 3 * (nv + 4) + 6 + 3
        noise = 3 * (ns + 1) + 6
        return {"bytes": 8 * cells * (state_in + npv + 3 + coef + flux + noise), "flops": cells * _step_flops(p) / 3}
    if kind == "stats":
        stats = 2 * nv + (npv + 3) + (npv + 5) + 26 + 2 * (nv + 1) + 12
        return {"bytes": 8 * cells * (nv + npv + 3 + 2 * stats), "flops": cells * 450}
    nvar, pairs, samples = len(SF_NAMES), SF_PAIRS, case["samples"]
    fft = 2.5 * nvar * math.log2(cells) * samples
    return {"bytes": 8 * cells * (nvar * samples + 3 * pairs), "flops": cells * (fft + 8 * pairs * samples + 8 * pairs)}


def tolerance(case):
    """About four times what a pass differs from ``exact``: FP64 steps 2.5e-7 (the in-kernel noise is formed in
    FP32), mixed steps up to 7e-5 (their coefficients and dissipative fluxes are FP32), the structure factor's
    imaginary parts 1.2e-12 (sums that nearly cancel), operators and statistics at FP64 rounding."""
    if case["kind"] in ("steps", "full", "ensemble"):
        return {"rel": 3e-4, "max": 3e-2} if case.get("mixed") else {"rel": 1e-6, "max": 1e-4}
    return {"rel": 1e-11, "max": 1e-8}


# ---- the same in plain torch, 64 bits ------------------------------------------------------

GH = 2                       # ghost layers
UNIT = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
EDGE_DIRS = ((0, 1), (0, 2), (1, 2))
MASK = 0xFFFFFFFF


def _win(a, lo, size):
    """The points lo .. lo + size - 1 (box indices) of an array with GH ghost layers."""
    for d in range(3):
        a = a.narrow(-1 - d, lo[d] + GH, size[d])
    return a


def _mulhilo(c, x):
    """High and low 32 bits of c * x for 32-bit unsigned values in int64."""
    low = (x & 0xFFFF) * c
    high = (x >> 16) * c + (low >> 16)
    return high >> 16, ((high & 0xFFFF) << 16) | (low & 0xFFFF)


def _philox_normals(point, pair, step, seed):
    """The two Box-Muller pairs ((z_A, z_B) of field 2q and of 2q + 1) of Philox-4x32-10, in 64 bits."""
    c = [point, torch.full_like(point, pair), torch.full_like(point, step & MASK), torch.full_like(point, step >> 32)]
    k0, k1 = seed & MASK, (seed >> 32) & MASK
    for _ in range(10):
        h0, l0 = _mulhilo(0xD2511F53, c[0])
        h1, l1 = _mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & MASK, (k1 + 0xBB67AE85) & MASK
    out = []
    for w0, w1 in ((c[0], c[1]), (c[2], c[3])):
        u1 = ((w0 >> 8).double() + 0.5) / 16777216.0
        u2 = ((w1 >> 8).double() + 0.5) / 16777216.0
        r = torch.sqrt(-2.0 * torch.log(u1))
        a = 2.0 * math.pi * (u2 - 0.5)
        out.append((r * torch.cos(a), r * torch.sin(a)))
    return out


def _solve(a, b, n):
    """Elementwise Gaussian elimination of the n x n systems a x = b."""
    a, b = [list(r) for r in a], list(b)
    for j in range(n - 1):
        for i in range(j + 1, n):
            f = a[i][j] / a[j][j]
            a[i] = [a[i][k] - f * a[j][k] for k in range(n)]
            b[i] = b[i] - f * b[j]
    for i in range(n - 1, -1, -1):
        b[i] = (b[i] - sum(a[i][j] * b[j] for j in range(i + 1, n))) / a[i][i]
    return b


class _Box:
    """One box of the staggered scheme on whole grown arrays (component, z, y, x)."""

    def __init__(self, p, fluct):
        self.p, self.n, self.ns = p, p.n_cells, p.nspecies
        self.wx = _wall_x(p)
        self.hcv, self.hcp = p.hc()
        self.dv = p.dx[0] * p.dx[1] * p.dx[2]
        rho_k, temp, mom = fluct
        rho, energy = _conserved(p, rho_k, temp, mom)
        self.cu, self.prim = self.new(p.nvars), self.new(p.nprimvars)
        self.mom, self.vel = [self.new(1, FACE[d]) for d in range(3)], [self.new(1, FACE[d]) for d in range(3)]
        hcv = sum(p.rhobar[k] * self.hcv[k] for k in range(self.ns))
        self.cu[0], self.cu[4] = p.rho0, p.rho0 * hcv * p.T_init
        for k in range(self.ns):
            self.cu[5 + k] = p.rho0 * p.rhobar[k]
        self.valid(self.cu[0]).copy_(rho)
        self.valid(self.cu[4]).copy_(energy)
        for k in range(self.ns):
            self.valid(self.cu[5 + k]).copy_(rho_k[k])
        for d in range(3):
            self.valid(self.mom[d][0], FACE[d]).copy_(mom[d])
        self.finish()

    def new(self, comps, nodal=CELL, ng=GH):
        shape = (comps,) + tuple(self.n[d] + nodal[d] + 2 * ng for d in (2, 1, 0))
        return torch.zeros(shape, dtype=torch.float64, device=_device())

    def valid(self, a, nodal=CELL):
        return _win(a, (0, 0, 0), [self.n[d] + nodal[d] for d in range(3)])

    def fill(self, a, nodal=CELL):
        for d in range(3):
            if d == 0 and self.wx:
                continue
            ax, n, e = -1 - d, self.n[d], nodal[d]
            a.narrow(ax, 0, GH).copy_(a.narrow(ax, n, GH).clone())
            a.narrow(ax, n + e + GH, GH).copy_(a.narrow(ax, GH + e, GH).clone())

    def convert(self):
        p, ns, n = self.p, self.ns, self.n
        for d in range(3):
            size = [n[q] + UNIT[d][q] for q in range(3)]
            lo = [-x for x in UNIT[d]]
            rho = _win(self.cu[0], lo, size) + _win(self.cu[0], (0, 0, 0), size)
            self.valid(self.vel[d][0], FACE[d]).copy_(2 * self.valid(self.mom[d][0], FACE[d]) / rho)
        cu = self.valid(self.cu)
        rho, out = cu[0], self.valid(self.prim)
        out[0] = rho
        kin = 0.0
        for d in range(3):
            v, m = self.valid(self.vel[d][0], FACE[d]), self.valid(self.mom[d][0], FACE[d])
            out[1 + d] = 0.5 * (_lo(v, d) + _hi(v, d))
            cu[1 + d] = 0.5 * (_lo(m, d) + _hi(m, d))
            kin = kin + (_lo(m, d) + _hi(m, d)) ** 2
        energy = (cu[4] - 0.125 * kin / rho) / rho
        y = [cu[5 + k] / rho for k in range(ns)]
        yf = [v.clamp(0.0, 1.0) for v in y]
        tot = sum(yf)
        cv = sum(yf[k] / tot * self.hcv[k] for k in range(ns))
        e0 = sum(yf[k] / tot * p.e0[k] for k in range(ns))
        out[4] = (energy - e0) / cv
        mix = 1.0 / sum(y[k] / p.molmass[k] for k in range(ns))
        out[5] = rho * p.Runiv / mix * out[4]
        for k in range(ns):
            out[6 + k] = y[k]
            out[6 + ns + k] = y[k] * mix / p.molmass[k]

    def walls(self):
        """setBCStag for impermeable x walls."""
        p, n, ns = self.p, self.n[0], self.ns
        for side in range(2):
            bc_vel, bc_therm = (p.bc_vel_lo, p.bc_vel_hi)[side][0], (p.bc_therm_lo, p.bc_therm_hi)[side][0]
            wall_t = (p.t_lo, p.t_hi)[side][0]
            ghost = [1, 0] if side == 0 else [n + GH, n + GH + 1]
            mirror = [GH, GH + 1] if side == 0 else [n + GH - 1, n + GH - 2]
            for f in (self.mom, self.vel):
                wall = f[0][..., :GH + 1] if side == 0 else f[0][..., n + GH:]
                wall.zero_()
                for d in (1, 2):
                    for a, b in zip(ghost, mirror):
                        f[d][..., a] = f[d][..., b] if bc_vel == 1 else 0.0
            for a, b in zip(ghost, mirror):
                self.prim[4:, ..., a] = self.prim[4:, ..., b]
                if bc_therm == 2:
                    self.prim[4, ..., a] = wall_t
                t, pr = self.prim[4, ..., a], self.prim[5, ..., a]
                y = [self.prim[6 + k, ..., a] for k in range(ns)]
                mix = 1.0 / sum(y[k] / p.molmass[k] for k in range(ns))
                rho = pr / (p.Runiv / mix) / t
                energy = sum(y[k] * (p.e0[k] + self.hcv[k] * t) for k in range(ns))
                kin = (self.mom[0][0, ..., a] + self.mom[0][0, ..., a + 1]) ** 2
                for d in (1, 2):
                    m = self.mom[d][0, ..., a]
                    kin = kin + (_lo_line(m, d) + _hi_line(m, d)) ** 2
                self.prim[0, ..., a] = self.cu[0, ..., a] = rho
                for k in range(ns):
                    self.cu[5 + k, ..., a] = rho * y[k]
                self.cu[4, ..., a] = rho * energy + 0.125 * kin / rho

    def finish(self):
        """FillBoundary, conversion, FillBoundary, setBCStag: what follows new conserved fields."""
        for d in range(3):
            self.fill(self.mom[d], FACE[d])
        self.fill(self.cu)
        self.convert()
        self.fill(self.cu)
        self.fill(self.prim)
        for d in range(3):
            self.fill(self.vel[d], FACE[d])
        if self.wx:
            self.walls()

    def transport(self):
        """Giovangigli's model on every grown cell."""
        p, ns, pi, kb = self.p, self.ns, math.pi, self.p.k_B
        rho, t, pr = self.prim[0], self.prim[4], self.prim[5]
        m = [p.molmass[k] * (kb / p.Runiv) for k in range(ns)]
        y = [self.prim[6 + k].clamp(0.0, 1.0) for k in range(ns)]
        tot = sum(y)
        y = [v / tot for v in y]
        mbar = 1.0 / sum(y[k] / m[k] for k in range(ns))
        x = [y[k] * mbar / m[k] for k in range(ns)]
        xsum = sum(x)
        x = [v + 1e-16 * (xsum / ns - v) for v in x]
        y = [x[k] * m[k] / mbar for k in range(ns)]
        diam = [[0.5 * (p.diameter[i] + p.diameter[j]) for j in range(ns)] for i in range(ns)]
        mu = [[m[i] * m[j] / (m[i] + m[j]) for j in range(ns)] for i in range(ns)]
        dbin = [[3.0 / 16.0 * torch.sqrt(2 * pi * (kb * t) ** 3 / mu[i][j]) / (pr * pi * diam[i][j] ** 2)
                 for j in range(ns)] for i in range(ns)]
        a = [[None] * ns for _ in range(ns)]
        for i in range(ns):
            eta1 = 5.0 / (16.0 * diam[i][i] ** 2) * torch.sqrt(m[i] * kb * t / pi)
            a[i][i] = x[i] * x[i] / eta1
            for k in range(ns):
                if k != i:
                    f = 2.0 * kb * t * x[i] * x[k] / (pr * dbin[i][k] * (m[i] + m[k]))
                    a[i][i] = a[i][i] + f * (1.0 + 0.6 * m[k] / m[i])
                    a[i][k] = f * (0.6 - 1.0)
        eta = sum(x[i] * b for i, b in enumerate(_solve(a, x, ns)))
        for i in range(ns):
            a[i][i] = 2.0 * x[i] * x[i] / dbin[i][i]
            for k in range(ns):
                if k != i:
                    f = x[i] * x[k] / dbin[i][k] * mu[i][k] / (m[i] + m[k])
                    a[i][i] = a[i][i] + f * (7.5 * m[i] / m[k] + 6.25 * m[k] / m[i] - 3.0 * m[k] / m[i] + 4.0)
                    a[i][k] = -f * (55.0 / 4.0 - 7.0)
        b = _solve(a, [2.5 * v for v in x], ns)
        kappa = sum(2.5 * x[i] * b[i] for i in range(ns)) * pr / t
        chi = []
        for i in range(ns):
            c = torch.zeros_like(t)
            for k in range(ns):
                if k != i:
                    f = 0.5 * x[k] / dbin[i][k] / (m[i] + m[k])
                    c = c + f * m[i] * b[k] - f * m[k] * b[i]
            chi.append(c)
        if ns == 1:
            dif = [torch.zeros_like(t)]
        else:
            dif = [rho * v for v in self._diffusion(dbin, x, y)]
        return {"eta": eta, "zeta": torch.zeros_like(eta), "kappa": kappa, "chi": chi, "D": dif}

    def _diffusion(self, dbin, x, y):
        ns = self.ns
        rng = range(ns)
        di = [(1.0 - y[i]) / sum(x[j] / dbin[i][j] for j in rng if j != i) for i in rng]
        minv = [di[i] / x[i] for i in rng]
        pm = [[(1.0 if i == j else 0.0) - y[j] for j in rng] for i in rng]
        jm = [[None] * ns for _ in rng]
        for i in rng:
            for j in rng:
                if i == j:
                    z = x[i] / di[i] - sum(x[i] * x[k] / dbin[i][k] for k in rng if k != i)
                else:
                    z = x[i] * x[j] / dbin[i][j]
                jm[i][j] = minv[i] * z
        pj = [[sum(pm[i][k] * jm[k][j] for k in rng) for j in rng] for i in rng]
        m2 = [[sum(pm[i][k] * minv[k] * pm[j][k] for k in rng) for j in rng] for i in rng]
        dif = m2
        for _ in range(3):
            dif = [[sum(pj[i][k] * dif[k][j] for k in rng) + m2[i][j] for j in rng] for i in rng]
        return [dif[i][j] * y[i] for j in rng for i in rng]

    # -- noise ---------------------------------------------------------------------------
    def _points(self, lo, size):
        """Canonical point indices of the lattice lo .. lo + size - 1."""
        p, axes, span = self.p, [], []
        for d in range(3):
            i = torch.arange(lo[d], lo[d] + size[d], device=_device(), dtype=torch.int64)
            wall = d == 0 and self.wx
            axes.append(i + 1 if wall else i % p.n_cells[d])
            span.append(p.n_cells[d] + 2 if wall else p.n_cells[d])
        z, yy, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
        return x + span[0] * (yy + span[1] * z)

    def step_noise(self, step):
        """A and B of every field of one step: lists of (A, B)."""
        seed, n, s2 = self.p.seed, self.n, math.sqrt(2.0)

        def fields(lo, size, fids):
            pt, got = self._points(lo, size), {}
            for q in sorted({f >> 1 for f in fids}):
                got[q] = _philox_normals(pt, q, step, seed)
            return [got[f >> 1][f & 1] for f in fids]

        face = [fields((0, 0, 0), [n[q] + FACE[d][q] for q in range(3)], [16 * d + c for c in range(self.ns + 1)])
                for d in range(3)]
        edge = [fields((0, 0, 0), [n[q] + EDGE[e][q] for q in range(3)], [48 + e])[0] for e in range(3)]
        cen = [tuple(s2 * z for z in f) for f in fields((-1, -1, -1), [v + 2 for v in n], [51, 52, 53])]
        chem = fields((0, 0, 0), n, [56 + m for m in range(self.p.nreaction)])
        return face, edge, cen, chem

    # -- fluxes --------------------------------------------------------------------------
    def _ends(self, d, lo, hi, mean):
        """Faces on the x walls take the ghost-side cell's value instead of the mean."""
        if d == 0 and self.wx:
            mean = mean.clone()
            mean[..., 0], mean[..., -1] = lo[..., 0], hi[..., -1]
        return mean

    def _wall_factor(self, kind):
        """StochFluxStag's factors along x for a wall condition of type 1 (0) or 2 (sqrt 2)."""
        f = torch.ones(self.n[0] + 1, dtype=torch.float64, device=_device())
        for side, at in ((0, 0), (1, -1)):
            f[at] = 0.0 if kind[side] == 1 else math.sqrt(2.0)
        return f

    def fluxes(self, c, w, dt):
        """calculateFluxStag: face fluxes (conserved and heat / viscous / Dufour parts), edge and centre fluxes."""
        p, n, ns, wx = self.p, self.n, self.ns, self.wx
        dx, kb = p.dx, p.k_B
        amp = kb / self.dv / dt
        wface, wedge, wcen = w
        pr = self.prim
        # cells grown by 1
        lo, size = (-1, -1, -1), [v + 2 for v in n]
        eta, t = _win(c["eta"], lo, size), _win(pr[4], lo, size)
        fac = torch.sqrt(2.0 * amp * eta * t)
        trace = sum(wcen)
        cs = [fac * wcen[d] - fac * trace / 3.0 for d in range(3)]
        at = lambda a, e, o=lo, s=size: _win(a, [o[q] + e[q] for q in range(3)], s)  # noqa: E731
        grad = [(at(self.vel[d][0], UNIT[d]) - at(self.vel[d][0], (0, 0, 0))) / dx[d] for d in range(3)]
        div = sum(grad)
        cd = [2.0 * eta * grad[d] - 2.0 / 3.0 * eta * div for d in range(3)]
        cen = []
        for d in range(3):
            m, v = self.mom[d][0], self.vel[d][0]
            cen.append(cs[d] - cd[d] + 0.25 * (at(m, (0, 0, 0)) + at(m, UNIT[d])) * (at(v, (0, 0, 0)) + at(v, UNIT[d]))
                       + at(pr[5], (0, 0, 0)))
        # edges
        es, ed, edge = [], [], [None] * 6
        for e, (p1, p2) in enumerate(EDGE_DIRS):
            o, s = (0, 0, 0), [n[q] + EDGE[e][q] for q in range(3)]
            m1, m2 = [-v for v in UNIT[p1]], [-v for v in UNIT[p2]]
            m12 = [m1[q] + m2[q] for q in range(3)]
            g = lambda a, off=(0, 0, 0): at(a, off, o, s)  # noqa: E731
            et = c["eta"] * pr[4]
            lo1 = 0.5 * (g(et, m12) + g(et, m1)), 0.5 * (g(c["eta"], m12) + g(c["eta"], m1))
            hi1 = 0.5 * (g(et, m2) + g(et)), 0.5 * (g(c["eta"], m2) + g(c["eta"]))
            etat = self._ends(p1, lo1[0], hi1[0], 0.5 * (lo1[0] + hi1[0]))
            ei = self._ends(p1, lo1[1], hi1[1], 0.5 * (lo1[1] + hi1[1]))
            h1 = torch.full((s[p1],), dx[p1], dtype=torch.float64, device=_device())
            if p1 == 0 and wx:
                h1[0] = h1[-1] = 0.5 * dx[0]
            h1 = h1.view([-1 if 2 - q == p1 else 1 for q in range(3)])
            g1 = (g(self.vel[p1][0]) - g(self.vel[p1][0], m2)) / dx[p2]
            g2 = (g(self.vel[p2][0]) - g(self.vel[p2][0], m1)) / h1
            es.append(torch.sqrt(2.0 * amp * etat) * wedge[e])
            ed.append(ei * (g1 + g2))
            total = es[e] * self._wall_factor((p.bc_vel_lo[0], p.bc_vel_hi[0])) if p1 == 0 and wx else es[e]
            u_lo, u_hi = g(self.vel[p2][0], m1), g(self.vel[p2][0])
            n_lo, n_hi = g(self.mom[p2][0], m1), g(self.mom[p2][0])
            um, nm = (self._ends(p1, a, b, 0.5 * (a + b)) for a, b in ((u_lo, u_hi), (n_lo, n_hi)))
            a1 = 0.5 * (g(self.mom[p1][0], m2) + g(self.mom[p1][0])) * um
            a2 = nm * 0.5 * (g(self.vel[p1][0], m2) + g(self.vel[p1][0]))
            # fluxes x: {v, w}, y: {u, w}, z: {u, v}
            edge[{0: 2, 1: 4, 2: 5}[e]] = total - ed[e] + a1
            edge[{0: 0, 1: 1, 2: 3}[e]] = total - ed[e] + a2
        face = [self._face(d, c, wface[d], amp, dt, cs, cd, es, ed) for d in range(3)]
        return face, edge, cen

    def _face(self, d, c, w, amp, dt, cs, cd, es, ed):
        p, n, ns, wx = self.p, self.n, self.ns, self.wx and d == 0
        s = [n[q] + UNIT[d][q] for q in range(3)]
        m1 = [-v for v in UNIT[d]]
        g = lambda a, off=(0, 0, 0): _win(a, off, s)  # noqa: E731
        mean = lambda a: self._ends(d, g(a, m1), g(a), 0.5 * (g(a, m1) + g(a)))  # noqa: E731
        diff = lambda a: g(a) - g(a, m1)  # noqa: E731
        pr = self.prim
        h = torch.full((s[d],), p.dx[d], dtype=torch.float64, device=_device())
        if wx:
            h[0] = h[-1] = 0.5 * p.dx[0]
        h = h.view([-1 if 2 - q == d else 1 for q in range(3)])
        # stresses are held on the cells grown by 1 and on the valid edges
        cell = lambda a: (_cell1(a, m1, s), _cell1(a, (0, 0, 0), s))  # noqa: E731
        u = g(self.vel[d][0])
        sl, sh = cell(cs[d])
        dl, dh = cell(cd[d])
        vdiag = 0.5 * u * (sl + sh) - 0.5 * u * (dl + dh)
        stoch, det = 0.0, 0.0
        for e, dirs in enumerate(EDGE_DIRS):
            if d not in dirs:
                continue
            q = dirs[0] if dirs[1] == d else dirs[1]
            for off in (0, 1):
                pos = [off * v for v in UNIT[q]]
                vel = self.vel[q][0]
                a, b = g(vel, [pos[r] + m1[r] for r in range(3)]), g(vel, pos)
                vm = self._ends(d, a, b, 0.5 * (a + b))
                stoch = stoch + 0.5 * vm * es[e].narrow(-1 - q, off, s[q])
                det = det + 0.5 * vm * ed[e].narrow(-1 - q, off, s[q])
        if wx:
            stoch = stoch * self._wall_factor((p.bc_vel_lo[0], p.bc_vel_hi[0]))
        vshear = stoch - det
        heat = torch.sqrt(amp * 2.0 * mean(c["kappa"] * pr[4] * pr[4])) * w[0]
        if wx:
            heat = heat * self._wall_factor((p.bc_therm_lo[0], p.bc_therm_hi[0]))
        heat = heat - mean(c["kappa"]) * diff(pr[4]) / h
        spec, duf = [torch.zeros_like(u) for _ in range(ns)], torch.zeros_like(u)
        if ns > 1:
            spec, duf = self._species(g, m1, mean, diff, h, d, c, w, dt)
            if wx:
                for a in spec + [duf]:
                    a[..., 0] = 0.0
                    a[..., -1] = 0.0
        f0 = g(self.mom[d][0])
        f4 = 0.5 * (g(self.cu[4], m1) + g(self.cu[4]) + g(pr[5], m1) + g(pr[5])) * u + heat + vdiag + vshear + duf
        fs = [spec[k] + 0.5 * (g(self.cu[5 + k], m1) + g(self.cu[5 + k])) * u for k in range(ns)] if ns > 1 else [f0]
        return [f0, f4] + fs, [heat, vdiag, vshear, duf]

    def _species(self, g, m1, mean, diff, h, d, c, w, dt):
        p, ns, pr = self.p, self.ns, self.prim
        rng = range(ns)
        yl, yh = ([g(pr[6 + k], o).clamp(0.0, 1.0) for k in rng] for o in (m1, (0, 0, 0)))
        tl, th = sum(yl), sum(yh)
        yl, yh = [v / tl for v in yl], [v / th for v in yh]
        mix = 1.0 / sum(0.5 * (yl[k] + yh[k]) / p.molmass[k] for k in rng)
        dl, dh = ([g(v, o) for v in c["D"]] for o in (m1, (0, 0, 0)))
        a = [[0.5 * (dl[j * ns + i] * yl[j] + dh[j * ns + i] * yh[j] + dl[i * ns + j] * yl[i] + dh[i * ns + j] * yh[i])
              for j in rng] for i in rng]
        chol = [[None] * ns for _ in rng]
        for i in rng:
            piv = a[i][i] - sum(chol[i][k] ** 2 for k in range(i))
            on = piv > 0.0
            chol[i][i] = torch.sqrt(piv.clamp(min=0.0))
            for j in range(i + 1, ns):
                v = a[i][j] - sum(chol[i][k] * chol[j][k] for k in range(i))
                chol[j][i] = torch.where(on, v / chol[i][i].clamp(min=1e-300), torch.zeros_like(v))
        fw = torch.sqrt(p.k_B * mix / self.dv / (p.Runiv * dt))
        wien = [fw * sum(chol[i][j] * w[1 + j] for j in range(i + 1)) for i in rng]
        t, pm = mean(pr[4]), mean(pr[5])
        hk = [p.e0[k] + self.hcp[k] * t for k in rng]
        duf = sum((hk[k] + p.Runiv * t / p.molmass[k] * mean(c["chi"][k])) * wien[k] for k in rng)
        dk = []
        for k in rng:
            x = pr[6 + ns + k]
            soret = mean(c["chi"][k] * x) * diff(pr[4]) / h / t
            dk.append(diff(x) / h + (mean(x) - mean(pr[6 + k])) * diff(pr[5]) / h / pm + soret)
        fk = [-sum(mean(c["D"][j * ns + i]) * dk[j] for j in rng) for i in rng]
        for k in rng:
            # z faces: the reference takes chi(i, j, k) twice
            chi = g(c["chi"][k]) if d == 2 else mean(c["chi"][k])
            duf = duf + (hk[k] + p.Runiv * t * chi / p.molmass[k]) * fk[k]
        return [wien[k] + fk[k] for k in rng], duf

    # -- the step ------------------------------------------------------------------------
    def chemistry(self, w, dt):
        p, ns = self.p, self.ns
        pr = self.valid(self.prim)
        t, navo = pr[4], p.avogadro if p.avogadro > 0 else p.Runiv / p.k_B
        conc = [pr[6 + ns + k] * pr[5] / p.Runiv / t for k in range(ns)]
        src = [torch.zeros_like(t) for _ in range(ns)]
        for m in range(p.nreaction):
            a = p.rate_const[m] * torch.exp(-p.alpha_param[m] / p.Runiv * (1.0 / t - 1.0 / p.T0_chem))
            a = a * (t / p.T0_chem) ** p.beta_param[m]
            for k in range(ns):
                a = a * conc[k] ** p.stoich_R[m][k]
            a = a.clamp(min=0.0)
            rate = a + (torch.sqrt(a / navo) * w[m] / math.sqrt(dt * self.dv) if p.reaction_type == 1 else 0.0)
            for k in range(ns):
                src[k] = src[k] + p.molmass[k] * (p.stoich_P[m][k] - p.stoich_R[m][k]) * rate
        return src

    def step(self, dt, step):
        """RK3stepStag; returns the stage-3 coefficients, fluxes and source."""
        p, n, ns = self.p, self.n, self.ns
        r2, r3 = math.sqrt(2.0), math.sqrt(3.0)
        weights = ((2 * r2 + r3) / 5.0, (-4 * r2 + 3 * r3) / 5.0, (r2 - 2 * r3) / 10.0)
        nface, nedge, ncen, nchem = self.step_noise(step)
        comps = [0, 4] + [5 + k for k in range(ns)]
        u0 = [self.valid(self.cu[q]).clone() for q in comps]
        mom0 = [self.valid(self.mom[d][0], FACE[d]).clone() for d in range(3)]
        for stage in range(3):
            mixw = lambda ab, b=weights[stage]: ab[0] + b * ab[1]  # noqa: E731
            c = self.transport()
            w = ([[mixw(f) for f in fs] for fs in nface], [mixw(f) for f in nedge], [mixw(f) for f in ncen])
            src = self.chemistry([mixw(f) for f in nchem], dt) if p.nreaction else None
            face, edge, cen = self.fluxes(c, w, dt)
            a0, a1, fdt = ((1.0, 0.0, dt), (0.75, 0.25, 0.25 * dt), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0 * dt))[stage]
            new = []
            for q, comp in enumerate(comps):
                div = sum((_hi(face[d][0][q], d) - _lo(face[d][0][q], d)) / p.dx[d] for d in range(3))
                v = a0 * u0[q] + (a1 * self.valid(self.cu[comp]) if stage else 0.0) - fdt * div
                if src is not None and q >= 2:
                    v = v + fdt * src[q - 2]
                new.append(v)
            newm = []
            names = ((None, 2, 4), (0, None, 5), (1, 3, None))
            for d in range(3):
                s = [n[q] + UNIT[d][q] for q in range(3)]
                tot = 0.0
                for q in range(3):
                    if q == d:
                        tot = tot + (_cell1(cen[d], (0, 0, 0), s) - _cell1(cen[d], [-v for v in UNIT[d]], s)) / p.dx[d]
                    else:
                        e = edge[names[d][q]]
                        tot = tot + (_hi(e, q) - _lo(e, q)) / p.dx[q]
                newm.append(a0 * mom0[d] + (a1 * self.valid(self.mom[d][0], FACE[d]) if stage else 0.0) - fdt * tot)
            if self.wx:
                newm[0][..., 0] = 0.0
                newm[0][..., -1] = 0.0
            for q, comp in enumerate(comps):
                self.valid(self.cu[comp]).copy_(new[q])
            for d in range(3):
                self.valid(self.mom[d][0], FACE[d]).copy_(newm[d])
            self.finish()
        return c, face, edge, cen, src

    def outputs(self):
        return {"cu": self.cu, "mom": self.mom, "prim": self.prim, "vel": self.vel}

    def flux_outputs(self, c, face, edge, cen):
        ns, out = self.ns, []
        for cons, aux in face:
            zero = torch.zeros_like(cons[0])
            out.append(torch.stack([cons[0], zero, zero, zero, cons[1]] + cons[2:] + aux))
        return {"coef": [c["eta"][None], c["zeta"][None], c["kappa"][None], torch.stack(c["chi"]), torch.stack(c["D"])],
                "faceflux": out, "edgeflux": [e[None] for e in edge], "cenflux": [v[None] for v in cen]}


def _lo_line(m, d):
    """Low faces of the cells of an x plane (z, y) of a momentum that is nodal in y (1) or z (2)."""
    return m.narrow(2 - d, 0, m.shape[2 - d] - 1)


def _hi_line(m, d):
    return m.narrow(2 - d, 1, m.shape[2 - d] - 1)


def _cell1(a, off, size):
    """Window of an array on the cells grown by 1."""
    for q in range(3):
        a = a.narrow(-1 - q, 1 + off[q], size[q])
    return a


def _run_mean(old, new, steps):
    return (old * (steps - 1.0) + new) / steps


def _exact_stats(p, boxes, cross):
    """Running statistics over the given states, in the order of statsStag.cpp."""
    ns, nv, npv = p.nspecies, p.nvars, p.nprimvars
    hcv, _ = p.hc()
    b0 = boxes[0]
    s = {"cuMeans": b0.new(nv), "cuVars": b0.new(nv), "primMeans": b0.new(npv + 3), "primVars": b0.new(npv + 5),
         "coVars": b0.new(26, CELL, 0), "mom3": b0.new(nv + 1, CELL, 0), "mom4": b0.new(nv + 1, CELL, 0)}
    for d in range(3):
        for k in ("velMeans", "velVars", "cumomMeans", "cumomVars"):
            s[f"{k}{d}"] = b0.new(1, FACE[d], 0)
    cr = torch.zeros(p.n_cells[0], 40 + ns, dtype=torch.float64, device=_device()) if cross else None
    line = None
    for steps, b in enumerate(boxes, 1):
        upd = lambda a, v: a.copy_(_run_mean(a, v, steps))  # noqa: E731
        cm, pm, cv, pv = (b.valid(s[k]) for k in ("cuMeans", "primMeans", "cuVars", "primVars"))
        cu, pr = b.valid(b.cu), b.valid(b.prim)
        mom = [b.valid(b.mom[d][0], FACE[d]) for d in range(3)]
        mm = [s[f"cumomMeans{d}"][0] for d in range(3)]
        upd(s["cuMeans"][0], b.cu[0])
        rho = cm[0]
        for d in range(3):
            upd(mm[d], mom[d])
            cm[1 + d] = 0.5 * (_lo(mm[d], d) + _hi(mm[d], d))
            pm[1 + d] = cm[1 + d] / rho
            upd(pm[npv + d], pr[1 + d])
        upd(cm[4], cu[4])
        for k in range(ns):
            upd(cm[5 + k], cu[5 + k])
            pm[6 + k] = cm[5 + k] / rho
            upd(pm[6 + ns + k], pr[6 + ns + k])
        pm[0] = rho
        upd(pm[4], pr[4])
        pm[5] = rho * p.Runiv * sum(pm[6 + k] / p.molmass[k] for k in range(ns)) * pm[4]
        rl, dl = [], []
        for d in range(3):
            size = [p.n_cells[q] + UNIT[d][q] for q in range(3)]
            off = [-v for v in UNIT[d]]
            r = 0.5 * (_win(s["cuMeans"][0], off, size) + _win(s["cuMeans"][0], (0, 0, 0), size))
            u = 0.5 * (_win(b.cu[0], off, size) + _win(b.cu[0], (0, 0, 0), size))
            s[f"velMeans{d}"][0] = mm[d] / r
            rl.append(r)
            dl.append(u - r)
        b.fill(s["cuMeans"])
        b.fill(s["primMeans"])
        for d in range(3):
            dj = mom[d] - mm[d]
            upd(s[f"cumomVars{d}"][0], dj * dj)
            dvel = (dj - s[f"velMeans{d}"][0] * dl[d]) / rl[d]
            upd(s[f"velVars{d}"][0], dvel * dvel)
        v = [0.5 * (_lo(s[f"velMeans{d}"][0], d) + _hi(s[f"velMeans{d}"][0], d)) for d in range(3)]
        drho, de = cu[0] - rho, cu[4] - cm[4]
        drk = [cu[5 + k] - cm[5 + k] for k in range(ns)]
        dy = [(drk[k] - pm[6 + k] * drho) / rho for k in range(ns)]
        cvm = sum(hcv[k] * cm[5 + k] / rho for k in range(ns))
        q = cvm * pm[4] - 0.5 * sum(x * x for x in v)
        dj = [0.5 * (_lo(mom[d], d) + _hi(mom[d], d)) - 0.5 * (_lo(mm[d], d) + _hi(mm[d], d)) for d in range(3)]
        dv = [(dj[d] - v[d] * drho) / rho for d in range(3)]
        dg = sum(v[d] * dj[d] for d in range(3))
        dt = pr[4] - pm[4]
        upd(cv[0], drho * drho)
        upd(cv[4], de * de)
        for k in range(ns):
            upd(cv[5 + k], drk[k] ** 2)
            upd(pv[6 + k], dy[k] ** 2)
        for d in range(3):
            upd(cv[1 + d], dj[d] ** 2)
            upd(pv[1 + d], dv[d] ** 2)
        pv[0] = cv[0]
        for c, x in enumerate((dg * dg, dg * de, drho * de, drho * dg)):
            upd(pv[npv + c], x)
        g = pv[npv:npv + 4]
        upd(pv[npv + 4], (cv[4] + g[0] - 2 * g[1] + q * (q * cv[0] - 2 * g[2] + 2 * g[3])) / (cvm * rho) ** 2)
        upd(pv[4], dt * dt)
        z = ns - 1
        terms = [drho * dj[0], drho * dj[1], drho * dj[2], dj[0] * dj[1], dj[1] * dj[2], dj[0] * dj[2], drho * de,
                 dj[0] * de, dj[1] * de, dj[2] * de, drk[0] * drk[z], drho * dv[0], drho * dv[1], drho * dv[2],
                 dv[0] * dv[1], dv[1] * dv[2], dv[0] * dv[2], drho * dt, dv[0] * dt, dv[1] * dt, dv[2] * dt,
                 dy[0] * dy[z], dy[0] * dv[0], dy[z] * dv[0], drk[0] * dv[0], drk[z] * dv[0]]
        for c, x in enumerate(terms):
            upd(s["coVars"][c], x)
        for c, x in enumerate([drho] + dv + [de] + dy + [dt]):
            upd(s["mom3"][c], x ** 3)
            upd(s["mom4"][c], x ** 4)
        b.fill(s["cuVars"])
        b.fill(s["primVars"])
        if cross:
            lines = [x.mean(dim=(-1 - 1, -1 - 2)).T for x in (cu, cm, pr[1:5 + ns], pm[1:5 + ns])]
            line = _exact_cross(p, cr, lines, steps)
    out = dict(s)
    if cross:
        out["spatialCross"], out["dataSliceMeans_xcross"] = cr, line
    return out


def _exact_cross(p, s, lines, steps):
    """EvaluateSpatialCorrelations3D on the x lines; returns the entries at x*."""
    ns, z = p.nspecies, p.nspecies - 1
    hcv, _ = p.hc()
    cu, cm, pr, pm = lines

    def point(i):
        c = {"rho": cm[i, 0], "ux": pm[i, 0], "drho": cu[i, 0] - cm[i, 0], "dK": cu[i, 4] - cm[i, 4],
             "dT": pr[i, 3] - pm[i, 3], "dvx": pr[i, 0] - pm[i, 0]}
        c["dj"] = [cu[i, 1 + d] - cm[i, 1 + d] for d in range(3)]
        c["dr"] = [cu[i, 5 + k] - cm[i, 5 + k] for k in range(ns)]
        c["Y"] = [pm[i, 4 + k] for k in range(ns)]
        c["dY"] = [pr[i, 4 + k] - pm[i, 4 + k] for k in range(ns)]
        cv = sum(hcv[k] * cm[i, 5 + k] / cm[i, 0] for k in range(ns))
        c["ci"] = 1.0 / cv
        c["q"] = cv * pm[i, 3] - 0.5 * sum(pm[i, d] ** 2 for d in range(3))
        c["dG"] = sum(pm[i, d] * c["dj"][d] for d in range(3))
        return c

    x, h = point(p.cross_cell), point(slice(None))

    def upd(q, v):
        s[:, q] = _run_mean(s[:, q], v, steps)

    for q, v in enumerate((x["drho"] * h["drho"], x["dK"] * h["dK"], x["dj"][0] * h["dj"][0], x["dj"][1] * h["dj"][1],
                           x["dj"][2] * h["dj"][2], x["dj"][0] * h["drho"], x["dj"][0] * h["dr"][0],
                           x["dj"][0] * h["dr"][z], x["drho"] * h["dr"][0], x["drho"] * h["dr"][z],
                           x["dr"][0] * h["drho"], x["dr"][z] * h["drho"], x["dG"] * h["dG"], x["dG"] * h["dK"],
                           x["dK"] * h["dG"], x["drho"] * h["dK"], x["dK"] * h["drho"], x["drho"] * h["dG"],
                           x["dG"] * h["drho"])):
        upd(q, v)
    a = [s[:, q] for q in range(19)]
    rr, ux = x["rho"] * h["rho"], x["ux"]
    s[:, 19] = x["ci"] * h["ci"] / rr * (a[1] + a[12] - a[13] - a[14] + h["q"] * x["q"] * a[0] - x["q"] * a[15]
                                         - h["q"] * a[16] + x["q"] * a[17] + h["q"] * a[18])
    s[:, 20] = x["ci"] / x["rho"] * (a[16] - a[18] - x["q"] * a[0])
    s[:, 21] = (a[5] - ux * a[0]) / x["rho"]
    s[:, 22] = (a[6] - ux * a[8]) / x["rho"]
    s[:, 23] = (a[7] - ux * a[9]) / x["rho"]
    s[:, 24] = (a[6] - ux * a[8] - h["Y"][0] * a[5] + ux * h["Y"][0] * a[0]) / rr
    s[:, 25] = (a[7] - ux * a[9] - h["Y"][z] * a[5] + ux * h["Y"][z] * a[0]) / rr
    for q, v in enumerate((x["dT"] * h["dT"], x["dT"] * h["drho"], x["dT"] * h["dvx"], x["dvx"] * h["drho"],
                           x["dvx"] * h["dY"][0], x["dvx"] * h["dY"][z], x["dvx"] * h["dr"][0], x["dvx"] * h["dr"][z],
                           x["dY"][0] * h["dY"][0], x["dY"][z] * h["dY"][z], x["dY"][0] * h["dY"][z]), 26):
        upd(q, v)
    for k in range(ns):
        upd(37 + k, x["dr"][k] * h["dr"][k])
    upd(37 + ns, x["dr"][z] * h["dr"][0])
    for q, k, i, j in ((1, 0, 8, 10), (2, z, 9, 11)):
        # the reference applies the running average of these entries a second time
        dd = _run_mean(s[:, 37 + k], x["dr"][k] * h["dr"][k], steps)
        s[:, 37 + ns + q] = (dd - x["Y"][k] * a[i] - h["Y"][k] * a[j] + x["Y"][k] * h["Y"][k] * a[0]) / rr
    c = p.cross_cell
    row = [v for q in (0, 4, 1, 2, 3) for v in (cu[c, q], cm[c, q])] + [v for q in range(4) for v in (pr[c, q], pm[c, q])]
    for k in range(ns):
        row += [cu[c, 5 + k], cm[c, 5 + k], pr[c, 4 + k], pm[c, 4 + k]]
    return torch.stack(row)


def exact(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    if kind == "ensemble":
        flat = {"cu": [], "mom": [], "prim": [], "vel": []}
        for p in _member_params(case, seed):
            b = _Box(p, _fluctuations(p, g))
            for q in range(case["steps"]):
                b.step(stable_dt(p), q)
            for key, v in b.outputs().items():
                flat[key] += [a.reshape(-1) for a in (v if isinstance(v, list) else [v])]
        return {k: torch.cat(v) for k, v in flat.items()}
    p = _params(case, seed)
    dt = stable_dt(p)
    if kind == "structfact":
        cov = torch.zeros((SF_PAIRS,) + tuple(p.n_cells[d] for d in (2, 1, 0)), dtype=torch.complex128, device=_device())
        pairs = [(j, i) for i in range(len(SF_NAMES)) for j in range(i, len(SF_NAMES))]
        cells = p.n_cells[0] * p.n_cells[1] * p.n_cells[2]
        for _ in range(case["samples"]):
            f = torch.fft.fftn(_sf_variables(p, g), dim=(1, 2, 3)) / math.sqrt(cells)
            for c, (a, b) in enumerate(pairs):
                cov[c] += torch.conj(f[a]) * f[b]
        cov = cov / case["samples"]
        cov[:, 0, 0, 0] = 0.0
        cov = torch.roll(cov, [p.n_cells[d] // 2 for d in (2, 1, 0)], (1, 2, 3))
        return [cov.real.contiguous(), cov.imag.contiguous(), cov.abs()]
    fluct = _fluctuations(p, g)
    if kind == "stats":
        return _exact_stats(p, [_Box(p, fluct), _Box(p, _fluctuations(p, g))], case["cross"])
    b = _Box(p, fluct)
    if kind == "operators":
        c = b.transport()
        faces, edges, cens = _operator_noise(p, g)
        grown = []
        for w in cens:
            a = b.new(1)
            b.valid(a[0]).copy_(w)
            b.fill(a)
            grown.append(_win(a[0], (-1, -1, -1), [v + 2 for v in p.n_cells]))
        got = b.fluxes(c, ([list(f) for f in faces], edges, grown), dt)
        return {"prim": b.prim, "vel": b.vel, **b.flux_outputs(c, *got)}
    last = None
    for q in range(case["steps"] if kind == "steps" else 1):
        last = b.step(dt, q)
    out = b.outputs()
    if kind == "full":
        c, face, edge, cen, src = last
        source = b.new(p.nprimvars)
        for k in range(p.nspecies if src is not None else 0):
            b.valid(source[5 + k]).copy_(src[k])
        out.update(source=source, **b.flux_outputs(c, face, edge, cen))
    return out
