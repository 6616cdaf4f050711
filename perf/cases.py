"""Timed cases of the engine: what a RocfluMP host has it do, through the
package's public entry points (Region, Batch), over the range of sizes, mesh
kinds, schemes and precisions it is used with.

A case is a dict of plain values:
  call       "solve"     upload a state, advance `steps` time steps (graph replay), download
             "residual"  `steps` residual evaluations of the resident state, the last to the host
             "host"      one time step of a state that the host keeps (step_host)
             "batch"     `regions` independent tubes advanced together
             "parts"     one mesh cut into `regions` coupled regions
  mesh       "tube" (n x 2 x 2 hexes), "tet" (n^3 x 6 jittered tets), "box" (n^3 mixed elements)
  scheme, reconst, precision   names as in the tables below
  mach       shock Mach number of the tet box
"""
import functools

import numpy as np
import torch

from rocflupicl_gb300 import case as K
from rocflupicl_gb300 import engine as E
from rocflupicl_gb300 import mesh as M
from rocflupicl_gb300 import partition as P

SCHEMES = {"roe": K.DISCR_UPW_ROE, "hllc": K.DISCR_UPW_HLLC, "ausm+": K.DISCR_UPW_AUSMPLUS,
           "ausm+up": K.DISCR_UPW_AUSMPLUSUP}
RECONST = {"venkat": K.RECONST_LIM_VENKAT, "weno": K.RECONST_WENO_XYZ}
PRECISION = {"fp64": K.PREC_FP64, "mixed": K.PREC_MIXED, "split": K.PREC_SPLIT}
CFL = 0.5


def _case(name, call, mesh, n, scheme, precision, steps, reconst="venkat", regions=1, mach=2.0):
    c = dict(call=call, mesh=mesh, n=n, scheme=scheme, reconst=reconst, precision=precision,
             steps=steps, regions=regions, mach=mach)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one residual of a tube of a few hundred cells: the smallest call, launches and latency
        _case("residual-tube128-fp64-hllc", "residual", "tube", 128, "hllc", "fp64", 1),
        # the Sod tube of the verification runs (1000 x 2 x 2 cells, double precision)
        _case("sod1000-fp64-ausm", "solve", "tube", 1000, "ausm+", "fp64", 50),
        # the smallest request of the serving stream (10k cells)
        _case("tet12-mixed-hllc", "solve", "tet", 12, "hllc", "mixed", 50, mach=2.5),
        # an ordinary request, in the mode with a double-precision update
        _case("tet32-split-ausm", "solve", "tet", 32, "ausm+", "split", 20, mach=1.5),
        # the large shock box (12.6 M tets), the mode a production run uses
        _case("tet128-mixed-roe", "solve", "tet", 128, "roe", "mixed", 10),
        # the same physics in double precision, the mode that reproduces the reference
        _case("tet64-fp64-roe", "solve", "tet", 64, "roe", "fp64", 2),
        # repeated residuals of the mixed-element box, both precisions
        _case("box96-fp64-hllc", "residual", "box", 96, "hllc", "fp64", 5),
        _case("box96-mixed-ausm", "residual", "box", 96, "ausm+", "mixed", 100),
        # an ensemble of tubes of uneven size as one batch
        _case("tubes48-mixed-ausm", "batch", "tube", 16000, "ausm+", "mixed", 60, regions=48),
        # a partitioned mesh: four regions with a halo exchange after every stage
        _case("parts4-tet40-fp64-hllc", "parts", "tet", 40, "hllc", "fp64", 2, regions=4),
        # the reference's default reconstruction, with the flux of its input decks
        _case("weno-tet64-mixed-ausmup", "solve", "tet", 64, "ausm+up", "mixed", 10, reconst="weno"),
        # a host that keeps the state and hands it over for each step
        _case("host-tet80-mixed-roe", "host", "tet", 80, "roe", "mixed", 1),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    call = rng.choice(["solve", "solve", "solve", "residual", "host", "batch", "parts"])
    scheme = rng.choice(sorted(SCHEMES))
    precision = rng.choice(["fp64", "fp64", "mixed", "mixed", "split"])
    fp64 = precision == "fp64"
    reconst = "weno" if call in ("solve", "host") and rng.random() < 0.25 else "venkat"
    mach = round(rng.uniform(1.2, 3.0), 3)
    regions = 1
    if call == "batch":
        mesh, n, regions = "tube", log(800, 3000 if fp64 else 16000), rng.randint(3, 48)
        cells = 4.0 * n / 3 * regions
    elif call == "parts":
        mesh, n, regions = "tet", log(12, 32 if fp64 else 64), rng.randint(2, 6)
        cells = 8.0 * n ** 3
    else:
        mesh = rng.choice(["tube", "tet"] if call != "residual" else ["tube", "tet", "box"])
        if mesh == "tube":
            n = log(33, 20000 if fp64 else 125000)
            cells = 4.0 * n
        else:
            n = log(7, 40 if fp64 else 90)
            cells = 6.0 * n ** 3
    # milliseconds of a step, roughly, to keep a pass below the largest listed one
    ms = 3 * (0.02 + cells * (7.0 if fp64 else 0.4) * (1.5 if reconst == "weno" else 1.0) / 1e6)
    steps = max(1, min(50, int(50.0 / ms)))
    if call == "host":
        steps = 1
    return _case(None, call, mesh, n, scheme, precision, steps, reconst, regions, mach)


# ---- meshes and states -----------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _mesh(kind, n):
    """The mesh of a case: what a program reads once and keeps."""
    if kind == "tube":
        return M.box(M.HEX, n, 2, 2, hi=(1.0, 2.0 / n, 2.0 / n))
    if kind == "tet":
        return M.box(M.TET, n, n, n, jitter=0.1, seed=2024)
    return M.box(M.MIXED, n, n, n)


def _tube_sizes(case):
    """Tube lengths of a batch, log-uniform down to a thirtieth of the longest."""
    r = np.random.default_rng(11)
    top = case["n"]
    return [max(16, int(round(top * 30.0 ** -r.random()))) for _ in range(case["regions"])]


@functools.lru_cache(maxsize=1)
def _meshes(kind, n, sizes):
    return [M.box(M.HEX, k, 2, 2, hi=(1.0, 2.0 / k, 2.0 / k)) for k in sizes]


def _numerics(case):
    return K.Numerics(spaceDiscr=SCHEMES[case["scheme"]], reconst=RECONST[case["reconst"]],
                      precision=PRECISION[case["precision"]], venkatGuard=1, cfl=CFL)


def _tube_case(m, num, rng):
    x = m.cofg[:, 0]
    left = x < rng.uniform(0.3, 0.7)
    rl, pl = rng.uniform(0.8, 1.2, size=2)
    rr, pr = np.exp(rng.uniform(np.log(0.1), np.log(0.8), size=2))
    ul, ur = rng.uniform(-0.3, 0.3, size=2)
    z = np.zeros_like(x)
    cv = K.prim_to_cv(num, np.where(left, rl, rr), np.where(left, ul, ur), z, z,
                      np.where(left, pl, pr))
    return K.Case("tube", m, num, K.tube_bcs(2), cv, K.eos_dv(num, cv))


def _tet_case(m, num, rng, mach):
    """Planar shock into quiescent air with a lognormal density perturbation."""
    N = m.nCells
    r = 1.2 * np.exp(0.1 * rng.standard_normal(N))
    u, p = np.zeros(N), np.full(N, 1.0e5)
    r2, u2, p2 = K.rankine_hugoniot(mach, num.refGamma, 1.2, 1.0e5)
    post = m.cofg[:, 0] < 0.2
    r, u, p = np.where(post, r2, r), np.where(post, u2, u), np.where(post, p2, p)
    z = np.zeros(N)
    cv = K.prim_to_cv(num, r, u, z, z, p)
    return K.Case("tet", m, num, K.tube_bcs(2), cv, K.eos_dv(num, cv))


def _cases(case, seed):
    """The engine cases (one per region) of a timed case, from the seed."""
    num = _numerics(case)
    rng = np.random.default_rng(seed)
    if case["call"] == "batch":
        ms = _meshes(case["mesh"], case["n"], tuple(_tube_sizes(case)))
        return [_tube_case(m, num, rng) for m in ms]
    m = _mesh(case["mesh"], case["n"])
    if case["mesh"] == "tube":
        return [_tube_case(m, num, rng)]
    if case["mesh"] == "box":
        cv = K.prim_to_cv(num, *K.fourier_state(m.cofg, seed))
        return [K.Case("box", m, num, [K.PatchBC(K.BC_SLIPWALL, 2) for _ in range(6)], cv,
                       K.eos_dv(num, cv))]
    whole = _tet_case(m, num, rng, case["mach"])
    if case["call"] != "parts":
        return [whole]
    out = []
    for part in _parts(case["mesh"], case["n"], case["regions"]):
        g = part.global_cells
        out.append(K.Case("part%d" % part.iRegionGlobal, part, num, whole.bcs, whole.cv[g].copy(),
                          whole.dv[g].copy()))
    return out


@functools.lru_cache(maxsize=1)
def _parts(kind, n, regions):
    return P.partition(_mesh(kind, n), regions)


def prepare(case, seed):
    """Registered regions, and page-locked host arrays for their states."""
    cs = _cases(case, seed)
    s = {"case": case, "regions": [E.Region(c) for c in cs]}
    N = [c.mesh.nTot for c in cs]
    at = np.concatenate([[0], np.cumsum(N)])
    if case["call"] == "residual":
        return s
    pin = torch.cuda.is_available()
    s["cv0"], s["cv"], s["dv"] = (
        torch.empty((int(at[-1]), k), dtype=torch.float64, pin_memory=pin).numpy() for k in (5, 5, 3))
    s["at"] = at
    for c, a, b in zip(cs, at[:-1], at[1:]):
        s["cv0"][a:b] = c.cv
        s["cv"][a:b] = c.cv
    for r in s["regions"]:
        r.set_time(1.0)  # a continued run: every time step from the CFL condition
    if case["call"] in ("batch", "parts"):
        s["batch"] = E.Batch(s["regions"], coupled=case["call"] == "parts")
    return s


def run(state):
    case, regs = state["case"], state["regions"]
    k = case["steps"]
    if case["call"] == "residual":
        for _ in range(k - 1):
            regs[0].residual(to_host=False)
        return [regs[0].residual()]
    cv0, cv, dv, at = state["cv0"], state["cv"], state["dv"], state["at"]
    if case["call"] == "host":
        regs[0].step_host(cv, dv, CFL, 1.0)
        return [cv, dv]
    for r, a, b in zip(regs, at[:-1], at[1:]):
        r.upload(cv0[a:b])
        r.set_time(1.0)
    if case["call"] == "solve":
        regs[0].steps_graph(k, CFL, 1.0)
    else:
        state["batch"].steps_graph(k, CFL, 1.0)
        state["batch"].sync()
    for r, a, b in zip(regs, at[:-1], at[1:]):
        r.download_into(cv[a:b], dv[a:b])
    return [cv, dv]


def work(case):
    """Per stage: the state read and written, the stage history, the geometry
    and the connectivity, each once; per pass: the state in and out."""
    if case["call"] == "batch":
        ms = _meshes(case["mesh"], case["n"], tuple(_tube_sizes(case)))
    elif case["call"] == "parts":
        ms = _parts(case["mesh"], case["n"], case["regions"])
    else:
        ms = [_mesh(case["mesh"], case["n"])]
    nc = sum(m.nTot for m in ms)
    nf, nb = sum(m.nFaces for m in ms), sum(m.nBFaces for m in ms)
    mem = sum(m.nMembs for m in ms)
    s = 8 if case["precision"] == "fp64" else 4
    geo = nc * 10 * s + 4 * mem + nf * (8 + 7 * s) + nb * (4 + 7 * s)
    stages = case["steps"] * (1 if case["call"] == "residual" else 3)
    state = nc * 40 if case["call"] == "residual" else nc * (40 + 40 + 10 * s)
    ends = nc * 40 if case["call"] == "residual" else nc * (40 + 64)
    flops = 35 * mem + 300 * (nf + nb) + 450 * nc
    return {"bytes": stages * (geo + state) + ends, "flops": stages * flops}


# ---- the same results in 64 bits, by plain tensor arithmetic ------------------------

class _Exact:
    """One region: least-squares gradients, limiter or WENO weights, fluxes."""

    def __init__(self, c, dev):
        m, num = c.mesh, c.numerics

        def t(a, dt=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(a)).to(dev).to(dt)

        self.num, self.N, self.nA = num, m.nTot, m.nCells
        self.vol, self.x = t(m.vol), t(m.cofg)
        self.c1, self.c2 = (t(m.f2c[:, k], torch.int64) - 1 for k in (0, 1))
        self.nrm, self.fc = t(m.fn), t(m.fc)
        self.off, self.mem = t(m.c2cs_off, torch.int64), t(m.c2cs_mem, torch.int32)
        self.b = [(bc.bcType, t(p.bf2c, torch.int64) - 1, t(p.fn), t(p.fc))
                  for p, bc in zip(m.patches, c.bcs) if p.n > 0]
        self.g, self.R = num.gamma_gv, 8314.3 / num.gv[1]
        A = torch.zeros(self.N, 3, 3, dtype=torch.float64, device=dev)
        for _, _, d, w in self.members():
            A += (w * d)[:, :, None] * d[:, None, :]
        self.Ai = torch.linalg.inv(A)
        self.cv = t(c.cv)

    def members(self):
        """Per stencil position: members, presence, offset and 1/|offset|^2 (0 where absent)."""
        cnt = self.off[1:] - self.off[:-1]
        for k in range(int(cnt.max())):
            on = k < cnt
            i = self.mem[torch.where(on, self.off[:-1] + k, self.off[:-1])].long() - 1
            d = self.x[i] - self.x
            yield i, on, d, torch.where(on, 1.0 / (d * d).sum(1), 0.0)[:, None]

    def prim(self):
        r = self.cv[:, :1]
        u = self.cv[:, 1:4] / r
        p = (self.g - 1.0) * (self.cv[:, 4:] - 0.5 * r * (u * u).sum(1, keepdim=True))
        return torch.cat([r, u, p], 1)

    def gradients(self, q):
        S = torch.zeros(self.N, 5, 3, dtype=q.dtype, device=q.device)
        for i, _, d, w in self.members():
            S += (q[i] - q)[:, :, None] * (w * d)[:, None, :]
        G = torch.einsum("nvd,nde->nve", S, self.Ai)
        return self.weno(q, G) if self.num.reconst == K.RECONST_WENO_XYZ else self.venkat(q, G)

    def weno(self, q, G):
        s = 1.0 / (G * G + 1e-15)
        top, bot = s * G, s.clone()
        for i, on, _, _ in self.members():
            bot += torch.where(on[:, None, None], s[i], 0.0)
            top += torch.where(on[:, None, None], s[i] * G[i], 0.0)
        G = top / bot
        for v in (0, 4):  # density and pressure stay positive at every face
            bad = torch.zeros(self.N, dtype=torch.int32, device=q.device)
            ends = [(self.c1, self.fc), (self.c2, self.fc)] + [(c, fc) for _, c, _, fc in self.b]
            for c, fc in ends:
                neg = q[c, v] + (G[c, v] * (fc - self.x[c])).sum(1) <= 0
                bad.index_put_((c[neg],), torch.ones((), dtype=torch.int32, device=q.device))
            G[bad > 0, v] = 0.0
        return G

    def venkat(self, q, G):
        lo, hi = q.clone(), q.clone()
        for a, b in ((self.c1, self.c2), (self.c2, self.c1)):
            i = a[:, None].expand(-1, 5)
            lo.scatter_reduce_(0, i, q[b], "amin")
            hi.scatter_reduce_(0, i, q[b], "amax")
        lim = torch.ones_like(q)
        for c in (self.c1, self.c2):
            d2 = (G[c] * (self.x[c] - self.fc)[:, None, :]).sum(2)
            dm = torch.where(d2 > 0, (hi - q)[c], (lo - q)[c])
            e = self.vol[c][:, None]
            a = dm * dm + e
            term = (a * d2 + 2.0 * d2 * d2 * dm) / (
                d2 * (a + 2.0 * d2 * d2 + dm * d2) + 1e-12 * torch.sign(d2))
            lim.scatter_reduce_(0, c[:, None].expand(-1, 5), torch.where(d2 == 0, 1.0, term), "amin")
        return G * lim[:, :, None]

    def residual(self):
        q = self.prim()
        G = self.gradients(q)
        c1, c2 = self.c1, self.c2
        L = q[c1] + (G[c1] * (self.fc - self.x[c1])[:, None, :]).sum(2)
        Rt = q[c2] + (G[c2] * (self.fc - self.x[c2])[:, None, :]).sum(2)
        f = _flux(self.num, L, Rt, 1.0 / q[c1, 0], 1.0 / q[c2, 0], self.nrm[:, :3]) * self.nrm[:, 3:]
        rhs = torch.zeros_like(q)
        rhs.index_add_(0, c1, f)
        rhs.index_add_(0, c2, -f)
        for kind, c, fn, fc in self.b:
            S = q[c] + (G[c] * (fc - self.x[c])[:, None, :]).sum(2)
            n = fn[:, :3]
            if kind == K.BC_SLIPWALL:
                f = torch.cat([0 * S[:, :1], S[:, 4:] * n, 0 * S[:, :1]], 1)
            else:  # supersonic outflow: the interior state
                r, u, p = S[:, :1], S[:, 1:4], S[:, 4:]
                m = r * (u * n).sum(1, keepdim=True)
                e = p / (r * (self.g - 1.0)) + 0.5 * (u * u).sum(1, keepdim=True)
                f = torch.cat([m, m * u + p * n, m * (e + p / r)], 1)
            rhs.index_add_(0, c, f * fn[:, 3:])
        rhs[self.nA:] = 0.0
        return rhs

    def dt(self):
        q = self.prim()
        a = torch.sqrt(self.g * q[:, 4] / q[:, 0])
        c1, c2 = self.c1, self.c2
        s = torch.zeros_like(a)
        f = ((0.5 * ((q[c1, 1:4] + q[c2, 1:4]) * self.nrm[:, :3]).sum(1)).abs()
             + 0.5 * (a[c1] + a[c2])) * self.nrm[:, 3]
        s.index_add_(0, c1, f)
        s.index_add_(0, c2, f)
        for _, c, fn, _ in self.b:
            s.index_add_(0, c, ((q[c, 1:4] * fn[:, :3]).sum(1).abs() + a[c]) * fn[:, 3])
        return CFL * (self.vol / s)[:self.nA].min()

    def outputs(self):
        q = self.prim()
        T = q[:, 4] / (q[:, 0] * self.R)
        return self.cv, torch.stack([q[:, 4], T, torch.sqrt(self.g * self.R * T)], 1)


def _flux(num, L, Rt, il, ir, n):
    g = num.refGamma
    gc = num.refCp - num.refCp / g
    (rl, ul, pl), (rr, ur, pr) = ((S[:, :1], S[:, 1:4], S[:, 4:]) for S in (L, Rt))
    il, ir = il[:, None], ir[:, None]

    def dot(a, b):
        return (a * b).sum(1, keepdim=True)

    ql, qr = dot(ul, n), dot(ur, n)
    kl, kr = 0.5 * dot(ul, ul), 0.5 * dot(ur, ur)
    al, ar = torch.sqrt(g * pl / rl), torch.sqrt(g * pr / rr)
    Hl, Hr = num.refCp * pl / (rl * gc) + kl, num.refCp * pr / (rr * gc) + kr

    def join(m, mom, en):
        return torch.cat([m, mom, en], 1)

    if num.spaceDiscr in (K.DISCR_UPW_AUSMPLUS, K.DISCR_UPW_AUSMPLUSUP):
        af = 0.5 * (al + ar)
        ml, mr = ql / af, qr / af
        w = 0.1875

        def split(x, s):  # Mach and pressure polynomials of side s
            big = x.abs() > 1.0
            q = x * x - 1.0
            mach = torch.where(big, 0.5 * (x + s * x.abs()),
                               s * 0.25 * (x + s) ** 2 + s * 0.125 * q * q)
            pres = torch.where(big, 0.5 * (1.0 + s * torch.sign(x)),
                               0.25 * (x + s) ** 2 * (2.0 - s * x) + s * w * x * q * q)
            return mach, pres

        (mp, wl), (mm, wr) = split(ml, 1.0), split(mr, -1.0)
        mf, pf = mp + mm, wl * pl + wr * pr
        if num.spaceDiscr == K.DISCR_UPW_AUSMPLUSUP:
            bar = 0.5 * (ml * ml + mr * mr)
            mf = mf - num.ausmKp * torch.clamp(1.0 - num.ausmSigma * bar, min=0.0) * (pr - pl) / (
                0.5 * (rl + rr) * af * af)
            pf = pf - num.ausmKu * wl * wr * af * (rl + rr) * (qr - ql)
        a, b = af * torch.clamp(mf, min=0.0) * rl, af * torch.clamp(mf, max=0.0) * rr
        return join(a + b, a * ul + b * ur + pf * n, a * Hl + b * Hr)
    if num.spaceDiscr == K.DISCR_UPW_ROE:
        rh = torch.sqrt(rl * rr)
        wt = rl / (rl + rh)
        uh, Hh = wt * ul + (1.0 - wt) * ur, wt * Hl + (1.0 - wt) * Hr
        qh, sh = dot(uh, n), 0.5 * dot(uh, uh)
        ah = torch.sqrt((g - 1.0) * (Hh - sh))
        d = num.epsentr * (qh + ah).abs()

        def fix(x):
            x = x.abs()
            return torch.where(x > d, x, (x * x + d * d) / (2.0 * d))

        l1, l2, l5 = fix(qh - ah), fix(qh), fix(qh + ah)
        du, dp = ur - ul, pr - pl
        dq = dot(du, n)
        t1 = l1 * (dp - rh * ah * dq) / (2.0 * ah * ah)
        t5 = l5 * (dp + rh * ah * dq) / (2.0 * ah * ah)
        t2, t3 = l2 * (rr - rl - dp / (ah * ah)), l2 * rh
        diss = join(t1 + t2 + t5,
                    t1 * (uh - n * ah) + t2 * uh + t3 * (du - n * dq) + t5 * (uh + n * ah),
                    t1 * (Hh - qh * ah) + t2 * sh + t3 * (dot(uh, du) - qh * dq) + t5 * (Hh + qh * ah))
        cen = join(ql * rl + qr * rr, ql * rl * ul + qr * rr * ur + (pl + pr) * n,
                   ql * rl * Hl + qr * rr * Hr)
        return 0.5 * cen - 0.5 * num.dissFact * diss
    el, er = pl / (rl * (g - 1.0)) + kl, pr / (rr * (g - 1.0)) + kr
    w = torch.sqrt(rr / rl)
    us, qs = (ul + w * ur) / (1.0 + w), (ql + w * qr) / (1.0 + w)
    Hs = (el + il * pl + w * (er + ir * pr)) / (1.0 + w)
    a_s = torch.sqrt((g - 1.0) * (Hs - 0.5 * dot(us, us)))
    sl, sr = torch.minimum(ql - al, qs - a_s), torch.maximum(qr + ar, qs + a_s)
    sm = (rr * qr * (sr - qr) - rl * ql * (sl - ql) - pr + pl) / (rr * (sr - qr) - rl * (sl - ql))
    ps = pl + rl * (ql - sl) * (ql - sm)

    def star(s, r, u, q, p, e):
        m = (s - q) * r
        return join(sm * m, sm * (m * u + (ps - p) * n), sm * (m * e + ps * sm - p * q)) / (s - sm) \
            + join(0 * ps, ps * n, sm * ps)

    def side(r, u, q, p, e):
        return join(q * r, q * r * u + p * n, q * (r * e + p))

    f = torch.where(sm > 0, star(sl, rl, ul, ql, pl, el), star(sr, rr, ur, qr, pr, er))
    f = torch.where(sr < 0, side(rr, ur, qr, pr, er), f)
    return torch.where(sl > 0, side(rl, ul, ql, pl, el), f)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cs = _cases(case, seed)
    X = [_Exact(c, dev) for c in cs]
    if case["call"] == "residual":
        return [X[0].residual().cpu()]
    ark, grk = (8.0 / 15.0, 5.0 / 12.0, 0.75), (0.0, 17.0 / 25.0, 5.0 / 9.0)  # Wray's scheme
    by = {c.mesh.iRegionGlobal: k for k, c in enumerate(cs)}
    for _ in range(case["steps"]):
        dts = [x.dt() for x in X]
        if case["call"] == "parts":
            dts = [min(dts)] * len(X)
        old = [None] * len(X)
        for a, g in zip(ark, grk):
            for k, x in enumerate(X):
                rhs = x.residual()
                d = rhs if old[k] is None else rhs - g * old[k]
                x.cv = x.cv - (a * dts[k] / x.vol)[:, None] * d
                old[k] = rhs
            for k, c in enumerate(cs):  # received cells take their owners' state
                for b in c.mesh.borders:
                    j = by[b.iRegionGlobal]
                    send = cs[j].mesh.borders[b.iBorder - 1].icgSend
                    X[k].cv[torch.as_tensor(b.icgRecv.astype(np.int64) - 1, device=dev)] = \
                        X[j].cv[torch.as_tensor(send.astype(np.int64) - 1, device=dev)]
    out = [x.outputs() for x in X]
    return [torch.cat([o[0] for o in out]).cpu(), torch.cat([o[1] for o in out]).cpu()]
