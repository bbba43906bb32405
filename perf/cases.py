"""The performance cases of the SCALE-DG dynamics step: what a user of the library has it do.

Every case is one pass through a public entry point of ``fedg.lib`` (a time step of ``Context.update``, a tracer
step, one application of the numerical diffusion, one explicit plus one implicit tendency of FElib's operator
interface) on a flat cube with a hydrostatic base state:

* ``bubble``      the +2 K warm bubble at rest: 125 m elements, constant temperature (the p = 3 configuration);
* ``current``     the -15 K density current in a 10 m/s wind: 800 m elements (the p = 7 configuration);
* ``stratified``  +-0.1 K noise in a stably stratified 5 m/s wind: 100 x 100 x 200 m elements (the large one);
* ``advection``   the tracer advection test: 3 x 3 x 4 km elements, no gravity, a (-35, -40) m/s wind.

All start with three-dimensional wind and pressure perturbations, so that no field is zero.  The time steps are
stable ones, so a state can be stepped again and again.  ``exact`` restates each path in plain torch float64.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fe-project_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

GRAV, RDRY, CPDRY, P00 = 9.80616, 287.04, 1004.64, 1.0e5
CVDRY = CPDRY - RDRY
KAP = CPDRY / CVDRY
FP64, MIXED, PAIR = "fp64", "mixed", "pair"

# element widths, wind, base state and the time step at the order it is quoted for
FLOWS = {
    "bubble": dict(h=125.0, hz=125.0, u0=0.0, v0=0.0, base="constT", grav=GRAV),
    "current": dict(h=800.0, hz=800.0, u0=10.0, v0=0.0, base="constT", grav=GRAV),
    "stratified": dict(h=100.0, hz=200.0, u0=5.0, v0=-3.0, base="constBVFreq", grav=GRAV),
    "advection": dict(h=3000.0, hz=4000.0, u0=-35.0, v0=-40.0, base="constPT", grav=0.0),
}


def _case(name, kind, prec, flow, p, nx, ny, nz, **more):
    return dict(name=name, kind=kind, prec=prec, flow=flow, p=p, nx=nx, ny=ny, nz=nz, **more)


def listed():
    return [
        # the warm bubble as FElib runs it (HEVE, SSP-RK3), in the fast arithmetic: the smallest call, where
        # latency and launches count
        _case("heve_pair_p3_8x8x8", "heve", PAIR, "bubble", 3, 8, 8, 8),
        # the same in FElib's own FP64 arithmetic
        _case("heve_fp64_p3_8x8x8", "heve", FP64, "bubble", 3, 8, 8, 8),
        # the warm bubble with the vertically implicit scheme (the precision form of that configuration)
        _case("hevi_pair_p3_8x8x8", "hevi", PAIR, "bubble", 3, 8, 8, 8),
        # the density current at its full size
        _case("hevi_pair_p7_32x32x8", "hevi", PAIR, "current", 7, 32, 32, 8),
        # the stratified flow at its full size, the headline step: 134 million nodes
        _case("hevi_pair_p7_128x128x16", "hevi", PAIR, "stratified", 7, 128, 128, 16),
        # the explicit scheme at p = 7 on a ragged mesh
        _case("heve_pair_p7_45x37x13", "heve", PAIR, "stratified", 7, 45, 37, 13),
        # FElib's algorithm in FP64 on a slice of the density current, Newton to 1e-10
        _case("hevi_fp64_p7_16x16x8", "hevi", FP64, "current", 7, 16, 16, 8),
        # the FP32 mode on a slice of the stratified flow
        _case("hevi_mixed_p7_32x32x16", "hevi", MIXED, "stratified", 7, 32, 32, 16),
        # FElib's operator interface: one cal_tend_ex and one linearised cal_vi, as its own driver calls them
        _case("felib_calls_p7_12x10x8", "felib", FP64, "current", 7, 12, 10, 8),
        # the tracer advection test's step (FCT and TMAR on) in FP64
        _case("tracer_fp64_p3_20x20x5", "tracer", FP64, "advection", 3, 20, 20, 5),
        # a tracer on a slice of the stratified mesh, in the fast arithmetic
        _case("tracer_pair_p7_32x32x16", "tracer", PAIR, "stratified", 7, 32, 32, 16),
        # the numerical diffusion after the dynamics step
        _case("numdiff_pair_p7_32x32x16", "numdiff", PAIR, "stratified", 7, 32, 32, 16, nlap=1),
    ]


# (kind, precision): flows, orders, the range of nodes
RANGES = {
    ("heve", PAIR): (("bubble", "stratified"), (3, 7), 1.0e4, 2.0e7),
    ("heve", FP64): (("bubble", "stratified"), (2, 3, 4, 5, 6, 7), 1.0e4, 3.0e6),
    ("hevi", PAIR): (("bubble", "current", "stratified"), (3, 7, 7), 2.0e4, 1.2e8),
    ("hevi", FP64): (("bubble", "current", "stratified"), (2, 3, 4, 5, 6, 7), 2.0e4, 2.0e6),
    ("hevi", MIXED): (("bubble", "current", "stratified"), (3, 7), 2.0e4, 2.0e7),
    ("felib", FP64): (("current", "stratified"), (2, 3, 5, 7), 2.0e4, 1.0e6),
    ("tracer", FP64): (("advection", "stratified"), (2, 3, 5, 7), 2.0e4, 4.0e6),
    ("tracer", PAIR): (("advection", "stratified"), (3, 7), 2.0e4, 3.0e7),
    ("numdiff", FP64): (("current", "stratified"), (2, 3, 5, 7), 2.0e4, 2.0e6),
    ("numdiff", PAIR): (("current", "stratified"), (3, 7), 2.0e4, 2.0e7),
}


def draw(rng):
    kind, prec = rng.choice(sorted(RANGES))
    flows, orders, lo, hi = RANGES[kind, prec]
    flow, p = rng.choice(flows), rng.choice(orders)
    ne = math.exp(rng.uniform(math.log(lo), math.log(hi))) / (p + 1) ** 3
    nz = rng.randint(2, 16)
    nz = max(2, min(nz, int(ne / 9) or 2))
    nx = max(3, min(160, int(round(math.sqrt(ne / nz) * rng.uniform(0.6, 1.6)))))
    ny = max(3, min(160, int(round(ne / nz / nx))))
    c = dict(kind=kind, prec=prec, flow=flow, p=p, nx=nx, ny=ny, nz=nz)
    if kind == "numdiff":
        c["nlap"] = rng.choice((1, 1, 2))
    return c


# ------------------------------------------------------------------------------------------------
def _dt(case):
    f, p, explicit = FLOWS[case["flow"]], case["p"], case["kind"] == "heve"
    if case["kind"] == "tracer":
        return (2.0 if case["flow"] == "advection" else 0.1) * min(1.0, 9.0 / p ** 2 if case["flow"] == "advection" else 1.0)
    if case["flow"] == "bubble":
        return 0.02 * min(1.0, 9.0 / p ** 2) * (0.9 if p > 3 else 1.0)
    if case["flow"] == "current":
        return 0.04
    return 0.0025 if explicit else 0.005


def _numdiff(case):
    """Coefficient and time step of the numerical diffusion: a tenth of the explicit limit."""
    f = FLOWS[case["flow"]]
    lam = 4.0 / min(f["h"], f["hz"]) ** 2 * case["p"] ** 4
    return 0.1 / (1.0e-3 * lam ** case["nlap"]), 1.0e-3


def _legendre(m, x):
    return np.polynomial.legendre.legval(x, [0.0] * m + [1.0])


def _nodes(p):
    """Legendre-Gauss-Lobatto nodes: -1, 1 and the roots of P_p'."""
    d = np.polynomial.legendre.legder([0.0] * p + [1.0])
    r = np.sort(np.polynomial.legendre.legroots(d).real)
    for _ in range(3):
        r = r - np.polynomial.legendre.legval(r, d) / np.polynomial.legendre.legval(r, np.polynomial.legendre.legder(d))
    return np.concatenate([[-1.0], 0.5 * (r - r[::-1]), [1.0]])


def _base(flow, z):
    """DENS_hyd, PRES_hyd, potential temperature of the hydrostatic base state at heights z (300 K at the surface)."""
    f, t0 = FLOWS[flow], 300.0
    if f["base"] == "constT":
        pres = P00 * np.exp(-z * f["grav"] / (RDRY * t0))
        return pres / (RDRY * t0), pres, t0 * (P00 / pres) ** (RDRY / CPDRY)
    if f["base"] == "constPT":
        ps = 101325.0
        ex = (ps / P00) ** (RDRY / CPDRY) - f["grav"] / (CPDRY * t0) * z
        pt = np.full_like(z, t0)
    else:
        n2 = 1.0e-4
        pt = t0 * np.exp(n2 / f["grav"] * z)
        ex = 1.0 + f["grav"] ** 2 / (CPDRY * n2) * (1.0 / pt - 1.0 / t0)
    pres = P00 * ex ** (CPDRY / RDRY)
    return pres / (RDRY * ex * pt), pres, pt


class _Mesh:
    """Node coordinates and the level profiles; fields have the shape (nz, ny, nx, k, j, i)."""

    def __init__(self, case, device):
        f, p = FLOWS[case["flow"]], case["p"]
        self.p, self.n1 = p, p + 1
        self.nx, self.ny, self.nz = case["nx"], case["ny"], case["nz"]
        self.h, self.hz = f["h"], f["hz"]
        self.dom = (0.0, self.h * self.nx, 0.0, self.h * self.ny, 0.0, self.hz * self.nz)
        r = 0.5 * (_nodes(p) + 1.0)
        t = lambda a, shape: torch.from_numpy(np.ascontiguousarray(a.reshape(shape))).to(device)  # noqa: E731
        n1 = self.n1
        self.x = t((np.arange(self.nx)[:, None] + r) * self.h, (1, 1, self.nx, 1, 1, n1))
        self.y = t((np.arange(self.ny)[:, None] + r) * self.h, (1, self.ny, 1, 1, n1, 1))
        self.z1 = (np.arange(self.nz)[:, None] + r) * self.hz
        lev = (self.nz, 1, 1, n1, 1, 1)
        self.z = t(self.z1, lev)
        self.dens1, self.pres1, self.pt1 = _base(case["flow"], self.z1)
        self.therm1 = P00 / RDRY * (self.pres1 / P00) ** (CVDRY / CPDRY)
        self.dens, self.pres, self.therm, self.pt = (t(a, lev) for a in (self.dens1, self.pres1, self.therm1, self.pt1))
        self.shape = (self.nz, self.ny, self.nx, n1, n1, n1)

    def full(self, prof):
        """A level profile as a host field (elements, nodes)."""
        a = np.broadcast_to(prof.reshape(self.nz, 1, 1, self.n1, 1, 1), self.shape)
        return np.ascontiguousarray(a).reshape(self.nz * self.ny * self.nx, self.n1 ** 3)


def _state(case, m, seed):
    """DDENS, MOMX, MOMY, MOMZ, DRHOT and, for a tracer case, its mixing ratio."""
    f = FLOWS[case["flow"]]
    dev = m.z.device
    r = random.Random(int(seed))
    lx, ly, lz = m.dom[1], m.dom[3], m.dom[5]
    bell = lambda xc, yc, zc, rx, ry, rz: torch.sqrt(  # noqa: E731
        ((m.x - xc) / rx) ** 2 + ((m.y - yc) / ry) ** 2 + ((m.z - zc) / rz) ** 2).clamp(max=1.0).mul(math.pi).cos().add(1.0).mul(0.5)
    if case["kind"] == "tracer":
        # a steady, divergence-free mass flux: horizontally uniform, sheared in z
        s = 1.0 + 0.2 * m.z / lz * r.uniform(0.5, 1.0)
        zero = torch.zeros(m.shape, dtype=torch.float64, device=dev)
        q = [zero.clone(), (m.dens * f["u0"] * s).expand(m.shape).contiguous(), (m.dens * f["v0"] * s).expand(m.shape).contiguous(),
             zero.clone(), zero.clone()]
        return q, bell(r.uniform(0.3, 0.7) * lx, r.uniform(0.3, 0.7) * ly, 0.4 * lz, 0.25 * lx, 0.25 * ly, 0.4 * lz).contiguous()
    if case["flow"] == "stratified":
        g = torch.Generator(device=dev).manual_seed(int(seed))
        th = (torch.rand(m.shape, generator=g, dtype=torch.float64, device=dev) - 0.5) * 0.2 * (m.z < 500.0)
    else:
        amp, rel = (2.0, 0.35) if case["flow"] == "bubble" else (-15.0, 0.45)
        th = amp * bell(r.uniform(0.4, 0.6) * lx, r.uniform(0.4, 0.6) * ly, rel * lz, 0.25 * lx, 0.25 * ly, 0.3 * lz)
    def wave(vert):
        a = 0.0
        for _ in range(2):
            kx, ky, kz = r.randint(1, 2), r.randint(0, 2), r.randint(1, 2)
            ph = 2.0 * math.pi * (kx * m.x / lx + ky * m.y / ly + r.random())
            a = a + torch.sin(ph) * vert(math.pi * kz * m.z / lz) * r.uniform(0.3, 0.5)
        return a

    # the temperature perturbation, in a pressure field with waves of some 50 Pa
    pt = m.pt + th
    del th
    rhot = P00 / RDRY * (m.pres * (1.0 + 5.0e-4 * wave(torch.cos)) / P00) ** (CVDRY / CPDRY)
    dens = rhot / pt
    del pt
    q = [dens - m.dens, None, None, None, rhot - m.therm]

    q[1] = dens * (f["u0"] + wave(torch.cos))
    q[2] = dens * (f["v0"] + wave(torch.cos))
    q[3] = dens * (0.5 * wave(torch.sin))
    return [a.contiguous() for a in q], None


def _flat(m, a):
    return a.reshape(m.nz * m.ny * m.nx, m.n1 ** 3)


def prepare(case, seed):
    from fedg import cases as fc
    from fedg import lib as fl

    m = _Mesh(case, "cuda")
    f = FLOWS[case["flow"]]
    fcase = fc.Case("perf", case["p"], case["nx"], case["ny"], case["nz"], m.dom, "HEVE" if case["kind"] == "heve" else "HEVI",
                    dt=_dt(case), nsteps=1, base=f["base"], grav=f["grav"])
    ctx = fl.Context(fcase)
    ctx.set_base_state(m.full(m.dens1), m.full(m.pres1), m.full(m.therm1))
    q, tracer = _state(case, m, seed)
    q = [_flat(m, a) for a in q]
    s = dict(kind=case["kind"], ctx=ctx, q=q, dt=_dt(case), prec={FP64: fl.PREC_FP64, MIXED: fl.PREC_MIXED, PAIR: fl.PREC_PAIR}[case["prec"]],
             eqs=fl.HEVE if case["kind"] == "heve" else fl.HEVI)
    if case["kind"] == "hevi":
        # the Newton tolerance each arithmetic is used with
        s["newton"] = dict(max_iter=10, tol=1e-13 if case["prec"] == PAIR else 1e-10)
    if case["kind"] == "felib":
        s["dpres"] = ctx.drhot2pres(q[4])[1]
        s["qs"], s["impl"] = _step_input(case, seed, q), (1.0 - 1.0 / math.sqrt(2.0)) * s["dt"]
    if case["kind"] == "tracer":
        s["Q"] = _flat(m, tracer)
        s["aM"], s["aP"] = ctx.trc_alphdens_advtest(*q[:4])
    if case["kind"] == "numdiff":
        s["nlap"], (s["coef"], s["dt"]) = case["nlap"], _numdiff(case)
    return s


def _step_input(case, seed, q):
    """A stage input near the state (elements, nodes): what an explicit stage leaves, with jumps between the elements."""
    g = torch.Generator(device=q[0].device).manual_seed(int(seed) + 77)
    return [a * (1.0 + 2.0e-3 * (torch.rand(a.shape[0], 1, generator=g, dtype=torch.float64, device=a.device) - 0.5)) for a in q]


def run(state):
    s, ctx = state, state["ctx"]
    if s["kind"] == "heve":
        ctx.update(s["q"], 1, eqs=s["eqs"], prec=s["prec"], dt=s["dt"])
        return list(s["q"])
    if s["kind"] == "hevi":
        failed, _ = ctx.update(s["q"], 1, eqs=s["eqs"], prec=s["prec"], dt=s["dt"], **s["newton"])
        return list(s["q"]) + [failed]
    if s["kind"] == "felib":
        return ctx.cal_tend_ex(s["q"], s["eqs"], dpres=s["dpres"]) + ctx.cal_vi(s["qs"], s["q"], s["impl"], s["dt"])
    if s["kind"] == "tracer":
        q = s["q"]
        return ctx.trc_update(s["Q"], q[1:4], s["aM"], s["aP"], q[0], q[0], s["dt"], prec=s["prec"])
    ctx.numdiff_apply(s["q"], s["nlap"], s["coef"], s["coef"], s["dt"], prec=s["prec"])
    return list(s["q"])


def work(case):
    """Bytes: each field of the pass read once and written once.  Flops: the derivative and Lift contractions, the flux
    and Rusanov arithmetic, one linear solve per implicit stage (3 x 3 blocks per node along a column)."""
    n1 = case["p"] + 1
    n = case["nx"] * case["ny"] * case["nz"] * n1 ** 3
    faces = 6.0 / n1
    tend = 5 * (6 * n1 + 12) + 45 + faces * 90
    solve = 2 * (3 * n1) ** 3 / 3.0 / n1 + 4 * 2 * (3 * n1) ** 2 / n1 + 60
    if case["kind"] == "heve":
        return {"bytes": 80.0 * n, "flops": (3 * (tend + 30) + 5 * 6 * n1) * n}
    if case["kind"] == "hevi":
        return {"bytes": 80.0 * n, "flops": (3 * (tend + 60) + 2 * solve + 5 * 6 * n1) * n}
    if case["kind"] == "felib":
        return {"bytes": (6 + 5 + 10 + 5) * 8.0 * n, "flops": (tend + solve) * n}
    if case["kind"] == "tracer":
        return {"bytes": (6 + 2 * faces) * 8.0 * n, "flops": 3 * (6 * n1 + 12 + 40 + faces * 20) * n}
    return {"bytes": 80.0 * n, "flops": 5 * (case["nlap"] * 2 * (6 * n1 + 12) + 10) * n}


# ------------------------------------------------------------------------------------------------
# The same passes in plain torch float64.
class _Ops:
    def __init__(self, case, m):
        p, n1 = m.p, m.n1
        x = _nodes(p)
        V = np.stack([_legendre(k, x) * math.sqrt(k + 0.5) for k in range(n1)], 1)
        iV = np.linalg.inv(V)
        D = np.zeros((n1, n1))
        lp = _legendre(p, x)
        for i in range(n1):
            for j in range(n1):
                if i != j:
                    D[i, j] = lp[i] / (lp[j] * (x[i] - x[j]))
        D[0, 0], D[p, p] = -p * (p + 1) / 4.0, p * (p + 1) / 4.0
        sig = np.ones(n1)
        etac = 2.0 / 3.0
        for k in range(1, n1):
            if k / p > etac:
                sig[k] = math.exp(-36.0 * ((k / p - etac) / (1.0 - etac)) ** 16)
        cut = np.ones(n1)
        cut[p] = 0.0
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(m.z.device)  # noqa: E731
        self.D, self.F, self.T = t(D), t(V @ np.diag(sig) @ iV), t(V @ np.diag(cut) @ iV)
        Mi = V @ V.T
        self.lb, self.lt = t(Mi[:, 0]), t(Mi[:, p])
        w = 2.0 / (p * (p + 1) * lp ** 2)
        self.w3 = t(w[:, None, None] * w[None, :, None] * w[None, None, :])
        self.w2 = t(w[:, None] * w[None, :])
        self.m, self.E = m, (2.0 / m.h, 2.0 / m.h, 2.0 / m.hz)
        self.grav = FLOWS[case["flow"]]["grav"]
        self.J = m.h * m.h * m.hz / 8.0
        # element axis and node axis of x, y, z
        self.ax = ((2, 5), (1, 4), (0, 3))

    def along(self, M, a, d):
        """M applied along the node axis of direction d."""
        if d == 0:
            return a @ M.T
        if d == 1:
            return M @ a
        s = a.shape
        return (M @ a.reshape(*s[:4], -1)).reshape(s)

    def side(self, a, d, top):
        return a.select(self.ax[d][1], self.m.p if top else 0)

    def outside(self, a, d, top, flip=False):
        """The exterior face values: the neighbour's, periodic in x and y; at a lid the own ones (flip: with the sign changed)."""
        e = self.ax[d][0]
        o = torch.roll(self.side(a, d, not top), -1 if top else 1, e)
        if d == 2:
            i = self.m.nz - 1 if top else 0
            own = self.side(a, d, top).select(0, i)
            o.select(0, i).copy_(-own if flip else own)
        return o

    def lift(self, fb, ft, d):
        """The Lift of the face values below (-) and above (+) in direction d."""
        ax = self.ax[d][1]
        shp = [1] * 6
        shp[ax] = self.m.n1
        return self.lb.reshape(shp) * fb.unsqueeze(ax) + self.lt.reshape(shp) * ft.unsqueeze(ax)

    def lev(self, prof, d, top):
        """A level profile at the face nodes of direction d."""
        return prof.expand(self.m.nz, 1, 1, self.m.n1, self.m.n1, self.m.n1).select(self.ax[d][1], self.m.p if top else 0)

    def dpres(self, dr):
        # PRES - PRES_hyd without cancellation
        return self.m.pres * torch.expm1(KAP * torch.log1p(dr / self.m.therm))

    def explicit(self, q, hevi, dp=None):
        """The explicit tendency: HEVE, or its HEVI part (horizontal mass and heat fluxes, no vertical pressure gradient)."""
        m = self.m
        dp = self.dpres(q[4]) if dp is None else dp
        dens = q[0] + m.dens
        pt = (m.therm + q[4]) / dens
        vel = [q[1 + d] / dens for d in range(3)]
        cs = torch.sqrt(KAP * (m.pres + dp) / dens)
        out = [None] * 5
        for d in range(3):
            vert = hevi and d == 2
            faces = []
            for top in (False, True):
                sg = 1.0 if top else -1.0
                mn = (self.side(q[1 + d], d, top), self.outside(q[1 + d], d, top, flip=d == 2))
                vn = (self.side(vel[d], d, top), self.outside(vel[d], d, top, flip=d == 2))
                c = (self.side(cs, d, top), self.outside(cs, d, top))
                faces.append((sg, vn, mn, None if vert else torch.maximum(vn[0].abs() + c[0], vn[1].abs() + c[1])))
            for v in range(5):
                if vert and v in (0, 4):
                    continue
                flux = q[1 + d] if v == 0 else (q[1 + d] * pt if v == 4 else q[v] * vel[d] + (dp if v == 1 + d and not vert else 0.0))
                ends = []
                for top, (sg, vn, mn, al) in zip((False, True), faces):
                    sides = []
                    for k, get in enumerate((self.side, self.outside)):
                        flip = dict(flip=True) if k and d == 2 and v == 3 else {}
                        fl = mn[k] if v == 0 else (mn[k] * get(pt, d, top) if v == 4 else get(q[v], d, top, **flip) * vn[k])
                        if v == 1 + d and not vert:
                            fl = fl + get(dp, d, top)
                        sides.append(fl)
                    jump = self.outside(q[v], d, top, flip=d == 2 and v == 3) - self.side(q[v], d, top)
                    r = (sides[1] - sides[0]) * sg
                    ends.append(0.5 * self.E[d] * (r if al is None else r - al * jump))
                t = self.E[d] * self.along(self.D, flux, d) + self.lift(ends[0], ends[1], d)
                out[v] = -t if out[v] is None else out[v] - t
        if not hevi:
            out[3] = out[3] - self.grav * self.along(self.T, q[0], 2)
        return out

    # -- the vertical implicit operator --
    def frozen(self, q0):
        """The frozen wave speed on the faces below and above."""
        dens = q0[0] + self.m.dens
        a = (q0[3] / dens).abs() + torch.sqrt(KAP * (self.m.pres + self.dpres(q0[4])) / dens)
        return [torch.maximum(self.side(a, 2, top), self.outside(a, 2, top)) for top in (False, True)]

    def vertical(self, P, fr, fm, al, uv=True):
        """The operator from the state P, the heat flux fr and the pressure deviation fm (all linear)."""
        E = self.E[2]

        def part(flux, v, flip_flux, flip_v):
            ends = []
            for top, a in zip((False, True), al):
                jv = self.outside(v, 2, top, flip=flip_v) - self.side(v, 2, top)
                r = -a * jv
                if flux is not None:
                    r = r + (self.outside(flux, 2, top, flip=flip_flux) - self.side(flux, 2, top)) * (1.0 if top else -1.0)
                ends.append(0.5 * E * r)
            t = self.lift(ends[0], ends[1], 2)
            return -t if flux is None else -(E * self.along(self.D, flux, 2) + t)

        A = [part(P[3], P[0], True, False), None, None, part(fm, P[3], False, True), part(fr, P[4], True, False)]
        A[3] = A[3] - self.grav * self.along(self.T, P[0], 2)
        if uv:
            A[1], A[2] = part(None, P[1], False, False), part(None, P[2], False, False)
        return A

    def implicit(self, P, al):
        pot = (self.m.therm + P[4]) / (self.m.dens + P[0])
        return self.vertical(P, pot * P[3], self.dpres(P[4]), al)

    def linear(self, P0, al):
        """v -> A'(P0) v."""
        dens, rhot = self.m.dens + P0[0], self.m.therm + P0[4]
        pot = rhot / dens
        gp = KAP * (self.m.pres + self.dpres(P0[4])) / rhot
        return lambda v: self.vertical(v, pot * v[3] + (v[4] - pot * v[0]) / dens * P0[3], gp * v[4], al)

    def solve(self, qs, q0, c, newton):
        """Q - qs - c A(Q) = 0 (converged), or one Newton step from q0."""
        al = self.frozen(q0)
        P = list(q0)
        for _ in range(newton):
            lin = self.linear(P, al)
            b = [s + c * a - p for s, a, p in zip(qs, self.implicit(P, al), P)]
            d, first = list(b), None
            for _ in range(60):  # a fixed point: the vertical Courant numbers are well below one
                e = [x + c * y for x, y in zip(b, lin(d))]
                off = [float((x - y).abs().max()) for x, y in zip(e, d)]
                first, d = first or off, e
            if any(x > 1.0e-9 * y for x, y in zip(off, first)) and newton == 1:
                return None
            P = [p + x for p, x in zip(P, d)]
            if not all(bool(torch.isfinite(p).all()) for p in P):
                return None
        return P

    def filter(self, q):
        return [self.along(self.F, self.along(self.F, self.along(self.F, a, 0), 1), 2) for a in q]

    def step_heve(self, q, dt):
        e = lambda x: [a + dt * b for a, b in zip(x, self.explicit(x, False))]  # noqa: E731
        q1 = e(q)
        q2 = [0.75 * a + 0.25 * b for a, b in zip(q, e(q1))]
        return self.filter([a / 3.0 + 2.0 / 3.0 * b for a, b in zip(q, e(q2))])

    def step_hevi(self, q, dt):
        s2 = math.sqrt(2.0)
        g, dl, al = 1.0 - 1.0 / s2, 0.25 * s2, (3.0 + 2.0 * s2) / 6.0
        te = [self.explicit(q, True)]
        ti = [self.implicit(q, self.frozen(q))]
        Q = None
        for ae, ai in (((2.0 * g,), (g,)), ((1.0 - al, al), (dl, dl))):
            qs = [a + dt * sum(x * t[v] for x, t in list(zip(ae, te)) + list(zip(ai, ti))) for v, a in enumerate(q)]
            Q = self.solve(qs, q, g * dt, 3)
            if Q is None:
                return None
            te.append(self.explicit(Q, True))
            ti.append([(a - b) / (g * dt) for a, b in zip(Q, qs)])
        return self.filter([a + dt * sum(b * (te[k][v] + ti[k][v]) for k, b in enumerate((dl, dl, g))) for v, a in enumerate(q)])

    # -- tracer --
    def tracer(self, Q, q, dt):
        m = self.m
        dens = q[0] + m.dens
        vel = [q[1 + d] / dens for d in range(3)]
        faces = []  # direction, top, mass flux inside and outside, alpha dens inside and outside
        for d in range(3):
            for top in (False, True):
                sg, fl = (1.0 if top else -1.0), d == 2
                mn = [g * sg for g in (self.side(q[1 + d], d, top), self.outside(q[1 + d], d, top, flip=fl))]
                al = torch.maximum(self.side(vel[d], d, top).abs(), self.outside(vel[d], d, top).abs())
                faces.append((d, top, mn, al * self.side(dens, d, top), al * self.outside(dens, d, top)))

        def parts(Q):
            out = []
            for d, top, mn, aM, aP in faces:
                qM, qP = self.side(Q, d, top), self.outside(Q, d, top)
                nf = 0.5 * ((qP * mn[1] + qM * mn[0]) - aP * qP + aM * qM)
                out.append((nf, (nf * self.w2).sum((-1, -2), keepdim=True) * (self.J * self.E[d]), qM * mn[0]))
            return out

        def tend(Q, dtt):
            f = parts(Q)
            net = sum(s.clamp(min=0.0) for _, s, _ in f)
            mass = self.J * (self.w3 * dens * Q / dtt).sum((-1, -2, -3)).reshape(net.shape)
            R = (mass / (net + 1.0e-10)).clamp(0.0, 1.0)
            t = 0.0
            for d in range(3):
                ends = []
                for (dd, top, mn, aM, aP), (nf, s, own) in zip(faces, f):
                    if dd != d:
                        continue
                    e = self.ax[d][0]
                    RP = torch.roll(R, -1 if top else 1, e)
                    if d == 2:
                        i = m.nz - 1 if top else 0
                        RP.select(0, i).copy_(R.select(0, i))
                    ends.append(self.E[d] * (nf * torch.where(torch.signbit(s), RP, R) - own))
                t = t - self.E[d] * self.along(self.D, q[1 + d] * Q, d) - self.lift(ends[0], ends[1], d)
            return t

        v0 = Q * dens
        x = (v0 + dt * tend(Q, dt)) / dens
        x = (0.75 * v0 + 0.25 * (x * dens) + 0.25 * dt * tend(x, dt)) / dens
        x = (v0 / 3.0 + 2.0 / 3.0 * (x * dens) + 2.0 / 3.0 * dt * tend(x, dt)) / dens
        wd = self.w3 * dens
        a, b = (wd * x).sum((-1, -2, -3), keepdim=True), (wd * x.clamp(min=0.0)).sum((-1, -2, -3), keepdim=True)
        return a * self.J / (b * self.J + 1.0e-32) * x.clamp(min=0.0)

    # -- numerical diffusion --
    def diffuse(self, q, nlap, coef, dt):
        m = self.m
        q = list(q)
        sgn = 1.0 if (nlap + 1) % 2 == 0 else -1.0

        def grad(h, v, w, var, bc):
            out = []
            for d, a in ((0, h), (1, h), (2, v)):
                u = a * w
                b = (self.outside(u, d, False) - self.side(u, d, False)) * -1.0
                t = torch.zeros_like(b)
                if d == 2:  # the lids are centred; the reflected momentum jumps there
                    f = -2.0 if var == 3 and bc else 0.0
                    b.select(0, 0).copy_(-0.5 * f * self.side(u, d, False).select(0, 0))
                    t.select(0, m.nz - 1).copy_(0.5 * f * self.side(u, d, True).select(0, m.nz - 1))
                out.append(self.E[d] * (self.along(self.D, u, d) + self.lift(b, t, d)))
            return out

        def div(G, var, w, ch, cv):
            """The horizontal and vertical parts of div(c w G) with w the weight (None: 1)."""
            parts = []
            for d, c in ((0, ch), (1, ch), (2, cv)):
                u = G[d] if w is None else w * G[d]
                t = self.outside(u, d, True) - self.side(u, d, True)
                b = torch.zeros_like(t)
                if d == 2:
                    f = 0.0 if var == 3 else -2.0
                    b.select(0, 0).copy_(-0.5 * f * self.side(u, d, False).select(0, 0))
                    t.select(0, m.nz - 1).copy_(0.5 * f * self.side(u, d, True).select(0, m.nz - 1))
                parts.append(c * self.E[d] * (self.along(self.D, u, d) + self.lift(b, t, d)))
            return parts[0] + parts[1], parts[2]

        for var in (4, 3, 1, 2, 0):
            dens = q[0] + m.dens
            one = torch.ones_like(dens)
            G = grad(q[var], q[var], one if var == 0 else 1.0 / dens, var, True)
            for _ in range(1, nlap):
                lh, lv = div(G, var, None, 1.0, 1.0)
                G = grad(lh, lv, one, var, False)
            lh, lv = div(G, var, None if var == 0 else dens, sgn * coef, sgn * coef)
            q[var] = q[var] + dt * (lh + lv)
        return q


def exact(case, seed):
    n = case["nx"] * case["ny"] * case["nz"] * (case["p"] + 1) ** 3
    if n > 4.0e7:
        return None
    m = _Mesh(case, "cuda")
    o = _Ops(case, m)
    q, Q = _state(case, m, seed)
    flat = lambda x: [_flat(m, a.contiguous()) for a in x]  # noqa: E731
    if case["kind"] == "heve":
        return flat(o.step_heve(q, _dt(case)))
    if case["kind"] == "hevi":
        r = o.step_hevi(q, _dt(case))
        return None if r is None else flat(r) + [None]
    if case["kind"] == "felib":
        c = (1.0 - 1.0 / math.sqrt(2.0)) * _dt(case)
        qs = [a.reshape(m.shape) for a in _step_input(case, seed, [_flat(m, a) for a in q])]
        P = o.solve(qs, q, c, 1)
        return flat(o.explicit(q, True)) + ([None] * 5 if P is None else flat([(a - b) / c for a, b in zip(P, qs)]))
    if case["kind"] == "tracer":
        return flat([o.tracer(Q, q, _dt(case))])[0]
    coef, dt = _numdiff(case)
    return flat(o.diffuse(q, case["nlap"], coef, dt))
