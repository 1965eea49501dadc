"""The work whose speed matters to users of this framework, as measurable cases.

Each case is a dict of plain values; ``kind`` names the program it stands for:

* ``fused``      a run on the fused state (``Solver``): some steps, then the
                 macroscopic fields and both distributions are read back, as a run
                 does for its output and restart files
* ``percall``    a run that calls the reference's subroutines one by one
                 (``Solver(fused=False)``), FP32 or the FP64 build
* ``ensemble``   many small independent runs advanced together
* ``adjoint``    gradient of a probe misfit over the fused step
* ``adjoint_pc`` the same gradient over the per-call path
* ``slabs``      one domain cut into j tiles, halo planes exchanged every step
* ``turbulence`` the inflow-turbulence fields of the next levels

``exact`` restates each program in plain torch at 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from lbm_b200 import Lbm, Params, Solver
from lbm_b200.adjoint import FusedProbeProblem, ProbeProblem, initial_state
from lbm_b200.api import Ensemble
from lbm_b200.slabs import SlabTile, step_local

VISC = 1.0e-4          # the repository's workloads (lattice units)
SMAG = 0.15
AMPL = 1.0e-4
LEVELS = 8             # turbulence levels a run holds


# ---- the cases ---------------------------------------------------------------------

def _flow(kind, nx, ny, nz, nl, steps, storage="f32", ibnd=1, kbnd=12, solids="none", turb=False, **kw):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, nl=nl, steps=steps, storage=storage, ibnd=ibnd, kbnd=kbnd,
                solids=solids, turb=turb, **kw)


def listed():
    def named(name, case):
        return dict(case, name=name)
    return [
        # a run coupled to another program, which reads the fields after every step, on a
        # grid of the smallest kind: launches and latency
        named("coupled_q27_f32_40x32x24", _flow("fused", 40, 32, 24, 27, 1, solids="sphere", turb=True)),
        # flow past a sphere, the configuration the accuracy checks are made on
        named("sphere_q27_f32_128x64x64", _flow("fused", 128, 64, 64, 27, 20, solids="sphere")),
        # the large channel with inflow turbulence (the benchmark's grid)
        named("channel_q27_f32_512x256x256", _flow("fused", 512, 256, 256, 27, 10, turb=True)),
        # the city on the same grid in FP16-offset storage
        named("city_q27_f16_512x256x256", _flow("fused", 512, 256, 256, 27, 10, storage="f16", solids="city", turb=True)),
        # a periodic box of odd extents: one cell per thread, general ghost kernels
        named("box_q19_f32_201x150x97", _flow("fused", 201, 150, 97, 19, 10, ibnd=0, kbnd=0)),
        # host code that switches call by call, with solids and the turbulence slice
        named("percall_q27_f32_256x128x128", _flow("percall", 256, 128, 128, 27, 4, solids="city", turb=True)),
        # the same in double precision
        named("percall_q19_f64_192x96x96", _flow("percall", 192, 96, 96, 19, 4, storage="f64", solids="sphere")),
        # 64 members of uneven size (the benchmark's ensemble)
        named("ensemble_q19_f32_64", dict(kind="ensemble", members=64, nl=19, steps=16, storage="f32", lo=96, hi=192)),
        # gradients of the probe misfit: the benchmark's grid and checkpoint interval
        named("adjoint_q19_256x128x128", _flow("adjoint", 256, 128, 128, 19, 20, solids="sphere")),
        named("adjoint_percall_q19_128x64x64", _flow("adjoint_pc", 128, 64, 64, 19, 10, solids="sphere")),
        # four j tiles in one process
        named("slabs_q27_f32_256x128x128", _flow("slabs", 256, 128, 128, 27, 8, tiles=4)),
        # the fields of one inflow plane
        named("turbulence_256x256", dict(kind="turbulence", ny=256, nz=256, nrturb=100, fields=3)),
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, min(hi, step * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)))


def draw(rng):
    kind = rng.choice(["fused", "fused", "fused", "percall", "percall", "ensemble", "adjoint", "adjoint_pc", "slabs",
                       "turbulence"])
    nl = rng.choice([19, 27])
    if kind == "turbulence":
        return dict(kind=kind, ny=_log(rng, 24, 256), nz=_log(rng, 24, 256), nrturb=_log(rng, 10, 100),
                    fields=rng.choice([3, 4]))
    if kind == "ensemble":
        hi = _log(rng, 32, 192, 8)
        return dict(kind=kind, members=_log(rng, 4, 64), nl=nl, steps=rng.choice([4, 7, 16]),
                    storage=rng.choice(["f32", "f16"]), lo=max(16, hi // 2), hi=hi)
    nx, ny, nz = _log(rng, 24, 512), _log(rng, 16, 256), _log(rng, 16, 256)
    cap = 3_000_000 if kind.startswith("adjoint") else 12_000_000
    while nx * ny * nz > cap:
        nx, ny, nz = max(24, nx * 4 // 5), max(16, ny * 4 // 5), max(16, nz * 4 // 5)
    solids = rng.choice(["none", "sphere", "city"])
    kbnd = rng.choice([12, 12, 11, 22])
    if kind == "fused":
        box = rng.random() < 0.25
        return _flow(kind, nx, ny, nz, nl, rng.choice([1, 4, 10]), storage=rng.choice(["f32", "f32", "f16"]),
                     ibnd=0 if box else 1, kbnd=0 if box else kbnd, solids=solids, turb=not box and rng.random() < 0.5)
    if kind == "percall":
        return _flow(kind, nx, ny, nz, nl, rng.choice([1, 3, 4]), storage=rng.choice(["f32", "f64"]), kbnd=kbnd,
                     solids=solids, turb=rng.random() < 0.5)
    if kind == "slabs":
        tiles = rng.choice([2, 3, 4])
        return _flow(kind, nx + nx % 2, max(4, ny // tiles) * tiles, nz, nl, rng.choice([2, 5, 8]),
                     storage=rng.choice(["f32", "f16"]), kbnd=kbnd, solids=solids, tiles=tiles)
    return _flow(kind, nx, ny, nz, nl, rng.choice([5, 10, 16]), kbnd=kbnd, solids=solids)


# ---- inputs --------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _dtype(case):
    return torch.float64 if case.get("storage") == "f64" else torch.float32


def _velocity(nx, ny, nz, uin, g, dtype):
    """rho, u, v, w (ghosts zero): a mean flow, large smooth eddies and small noise."""
    def wave(n):
        x = torch.arange(1, n + 1, device="cuda", dtype=dtype) * (2 * math.pi / n)
        ph = torch.rand((), generator=g, device="cuda", dtype=dtype) * (2 * math.pi)
        return torch.sin(x + ph)
    out = [torch.zeros((nz + 2, ny + 2, nx + 2), dtype=dtype, device="cuda") for _ in range(4)]
    inner = (slice(1, nz + 1), slice(1, ny + 1), slice(1, nx + 1))
    out[0][inner] = 1.0
    for q in range(3):
        noise = (torch.rand((nz, ny, nx), generator=g, device="cuda", dtype=dtype) - 0.5) * 2.0e-3
        noise += (0.3 * uin) * wave(nz)[:, None, None] * wave(ny)[None, :, None] * wave(nx)[None, None, :]
        out[q + 1][inner] = noise + (uin if q == 0 else 0.0)
    return out


def _mask(case, g):
    """blanking: a sphere, or boxes standing on the bottom wall."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["solids"] == "none":
        return None
    m = torch.zeros((nz + 2, ny + 2, nx + 2), dtype=torch.int32, device="cuda")
    if case["solids"] == "sphere":
        k, j, i = (torch.arange(n + 2, device="cuda") for n in (nz, ny, nx))
        r = min(ny, nz) / 8.0
        d = (i[None, None, :] - nx // 4) ** 2 + (j[None, :, None] - ny // 2) ** 2 + (k[:, None, None] - nz // 2) ** 2
        return (d < r * r).to(torch.int32)
    for x, y, h in torch.rand((16, 3), generator=g, device="cuda").tolist():
        i0, j0 = 1 + int(x * 0.7 * nx) + nx // 8, 1 + int(y * 0.85 * ny)
        m[1:2 + int((0.05 + 0.2 * h) * nz), j0:j0 + max(2, ny // 10), i0:i0 + max(2, nx // 20)] = 1
    m[:, :, 0] = m[:, :, -1] = m[:, 0] = m[:, -1] = m[0] = m[-1] = 0
    return m


def _levels(ny, nz, g, dtype):
    """uu, vv, ww (LEVELS + 1, nz, ny): smooth fields of unit variance, correlated in time."""
    ky, kz = (torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) for n in (ny, nz))
    spec = torch.exp(-40.0 * math.pi * (ky[None, :] ** 2 + kz[:, None] ** 2))
    out = []
    for _ in range(3):
        a = torch.fft.ifft2(torch.randn((LEVELS + 1, nz, ny), generator=g, device="cuda", dtype=torch.float64) * spec).real
        for t in range(1, LEVELS + 1):
            a[t] = 0.98 * a[t - 1] + 0.2 * a[t]
        a -= a.mean(dim=(1, 2), keepdim=True)
        a /= a.std(dim=(1, 2), keepdim=True)
        out.append(a.to(dtype).contiguous())
    return out


def _inputs(case, seed):
    g, dt = _gen(seed), _dtype(case)
    uin = 0.05
    d = {"macro": _velocity(case["nx"], case["ny"], case["nz"], uin, g, dt)}
    z = torch.linspace(0.0, 1.0, case["nz"], device="cuda", dtype=dt)
    d["uvel"] = uin * (1.0 + 0.1 * torch.sin(math.pi * z))
    d["mask"] = _mask(case, g)
    d["turb"] = _levels(case["ny"], case["nz"], g, dt) if case["turb"] else None
    return d


def _probe_inputs(case, seed):
    """Initial f1, f2 away from exact equilibrium (where the eddy viscosity has no
    derivative), probes and their target velocities."""
    d = _inputs(case, seed)
    g = _gen(seed + 104729)
    nx, ny, nz, nl = case["nx"], case["ny"], case["nz"], case["nl"]
    with Lbm(_params(case)) as L:
        f1, f2 = initial_state(L, *d["macro"], d["uvel"])
        torch.cuda.synchronize()
    f1 *= 1.0 + 2.0e-3 * torch.randn(f1.shape, generator=g, device="cuda")
    n = 200
    cell = torch.randperm(nx * ny * nz, generator=g, device="cuda")[:n]
    d["probes"] = torch.stack([cell % nx + 1, (cell // nx) % ny + 1, cell // (nx * ny) + 1], dim=1).cpu().numpy()
    t = 0.02 * torch.randn((n, 3), generator=g, device="cuda")
    t[:, 0] += 0.06
    d.update(f1=f1, f2=f2, target=t)
    return d


def _members(case, seed):
    """Params-like dicts of the members: extents multiples of 8, drawn from the seed of
    the ensemble's own sizes (the same for every input seed), inflow from the input's."""
    rs = np.random.RandomState(case["members"] * 1000 + case["hi"])
    rv = np.random.RandomState(seed % (2 ** 31))
    out = []
    for _ in range(case["members"]):
        nx = 8 * int(rs.randint(case["lo"] // 8, case["hi"] // 8 + 1))
        ny, nz = (8 * int(rs.randint(max(2, case["lo"] // 16), max(2, case["hi"] // 16) + 1)) for _ in range(2))
        out.append(_flow("fused", nx, ny, nz, case["nl"], case["steps"], storage=case["storage"], turb=True,
                         uin=float(rv.uniform(0.03, 0.07)), seed=int(rv.randint(1 << 30))))
    return out


def _member_inputs(m):
    g = _gen(m["seed"])
    return {"macro": _velocity(m["nx"], m["ny"], m["nz"], m["uin"], g, torch.float32),
            "uvel": torch.full((m["nz"],), m["uin"], device="cuda"), "mask": None,
            "turb": _levels(m["ny"], m["nz"], g, torch.float32)}


def _params(case):
    return Params(nx=case["nx"], ny=case["ny"], nz=case["nz"], nl=case["nl"], ibnd=case["ibnd"], jbnd=0, kbnd=case["kbnd"],
                  iturb_pos=min(10, case["nx"]), storage="f16" if case["storage"] == "f16" else "f32", kinevisc=VISC,
                  smagorinsky=SMAG)


# ---- the programs ----------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("fused", "percall"):
        d = _inputs(case, seed)
        turb = None if d["turb"] is None else (*d["turb"], LEVELS, AMPL)
        s["solver"] = Solver(_params(case), *d["macro"], d["uvel"], blanking=d["mask"], turbulence=turb,
                             fused=kind == "fused")
    elif kind == "ensemble":
        mem = _members(case, seed)
        ens = Ensemble([_params(m) for m in mem])
        for L, m in zip(ens.members, mem):
            d = _member_inputs(m)
            f1, f2 = initial_state(L, *d["macro"], d["uvel"])
            L.state_import(f1, f2, *d["macro"])
            L.set_inflow(d["uvel"])
            L.set_turbulence(*d["turb"], LEVELS, AMPL)
        # one array per field for all members, each member's part a view of it
        cells = [(m["nz"] + 2) * (m["ny"] + 2) * (m["nx"] + 2) for m in mem]
        flat = [torch.empty(sum(cells), device="cuda") for _ in range(4)]
        parts = [[t.view(L.p.sshape) for L, t in zip(ens.members, f.split(cells))] for f in flat]
        s.update(ens=ens, flat=flat, parts=parts)
    elif kind in ("adjoint", "adjoint_pc"):
        d = _probe_inputs(case, seed)
        make = FusedProbeProblem if kind == "adjoint" else ProbeProblem
        s["problem"] = make(_params(case), d["probes"], case["steps"], blanking=d["mask"], checkpoint=10)
        s.update({k: d[k] for k in ("f1", "f2", "uvel", "target")})
    elif kind == "slabs":
        d = _inputs(case, seed)
        p = _params(case)
        with Lbm(p) as L:
            f1, f2 = initial_state(L, *d["macro"], d["uvel"])
            torch.cuda.synchronize()
        s["tiles"] = [SlabTile(p, r, case["tiles"]) for r in range(case["tiles"])]
        for t in s["tiles"]:
            t.import_global(f1, f2, *d["macro"])
            t.set_inflow(d["uvel"])
            if d["mask"] is not None:
                t.set_solids(d["mask"])
    else:
        s["lbm"] = Lbm(Params(nx=32, ny=case["ny"], nz=case["nz"], nl=19, iturb_pos=10))
        s["out"] = [torch.empty((case["nrturb"] + 1, case["nz"], case["ny"]), device="cuda") for _ in range(case["fields"])]
        s["seed"] = int(seed)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("fused", "percall"):
        sol = state["solver"]
        sol.step(case["steps"])
        rho, u, v, w = sol.macro()
        f1, f2 = sol.state()
        return {"rho": rho, "u": u, "v": v, "w": w, "f1": f1, "f2": f2}
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        for m, L in enumerate(state["ens"].members):
            L.get_macro(*(p[m] for p in state["parts"]))
        return dict(zip(("rho", "u", "v", "w"), state["flat"]))
    if kind in ("adjoint", "adjoint_pc"):
        pr = state["problem"]
        u = pr.forward(state["f1"], state["f2"], state["uvel"])
        g, guvel = pr.backward(u - state["target"])
        return {"u": u, "f1_grad": g, "uvel_grad": guvel}
    if kind == "slabs":
        step_local(state["tiles"], case["steps"])
        out = {}
        for r, t in enumerate(state["tiles"]):
            L = t.lbm
            m = [L.empty_s() for _ in range(4)]
            f = [L.empty_f() for _ in range(2)]
            L.get_macro(*m)
            L.state_export(*f)
            out.update({"%s_%d" % (n, r): x for n, x in zip(("rho", "u", "v", "w", "f1", "f2"), m + f)})
        return out
    o = state["out"]
    state["lbm"].inflow_turbulence_compute(o[0], o[1], o[2], case["nrturb"], state["seed"],
                                           rr=o[3] if case["fields"] == 4 else None)
    return list(o)


def work(case):
    kind = case["kind"]
    if kind == "turbulence":
        # the fields written once; per level a real 2-D transform and the chain
        n = case["fields"] * (case["nrturb"] + 1) * case["ny"] * case["nz"]
        return {"bytes": 4.0 * n, "flops": n * (2.5 * math.log2(case["ny"] * case["nz"]) + 10.0)}
    Q, n = case["nl"], case["steps"]
    el = {"f16": 2.0, "f32": 4.0, "f64": 8.0}[case.get("storage", "f32")]
    # about this many operations for one collision in the closed form
    flop = 430.0 if Q == 27 else 330.0
    if kind == "ensemble":
        cells = sum(m["nx"] * m["ny"] * m["nz"] for m in _members(case, 0))
        return {"bytes": cells * (n * 2 * Q * el + Q * el + 16.0), "flops": cells * n * flop}
    cells = float(case["nx"] * case["ny"] * case["nz"])
    if kind in ("fused", "slabs"):
        # a step reads and writes each population; the outputs: f1, f2 and the four fields
        # from the two buffers
        return {"bytes": cells * (n * 2 * Q * el + 2 * Q * el + 2 * Q * 4.0 + 16.0), "flops": cells * n * flop}
    # a per-call step: postcoll reads f, rho, u, v, w, writes f, tau; drift reads and writes f;
    # macrovars reads f, writes four fields
    percall = (5 * Q + 9) * el
    if kind == "percall":
        return {"bytes": cells * n * percall, "flops": cells * n * flop}
    if kind == "adjoint":
        # forward and replay steps; a reverse step reads the populations and the adjoint, writes the adjoint
        return {"bytes": cells * n * (2 * 2 * Q + 3 * Q) * 4.0, "flops": cells * n * (2 * flop + 800.0)}
    # forward and replay; per reverse step: drift and macrovars (read, write the adjoint, read eight
    # fields), collision (read f and the adjoint, write it, read four fields, write four)
    return {"bytes": cells * n * (2 * percall + (2 * Q + 8 + 3 * Q + 8) * 4.0), "flops": cells * n * (2 * flop + 800.0)}


def tolerance(case):
    """About four times what the outputs were measured to be from ``exact`` (or, for the
    gradients, the FP32 fused and per-call sweeps from each other) over these ranges: the
    transverse velocities are the worst, the populations ten times better."""
    kind = case["kind"]
    if kind == "turbulence":
        return {"rel": 3.0e-6}           # measured 6e-7
    if kind.startswith("adjoint"):
        return {"rel": 2.0e-5}           # measured 1e-6 from exact; near tau's kink up to 5e-6
    if case["storage"] == "f64":
        return {"rel": 4.0e-14}          # measured 8e-15
    if case["storage"] == "f16":
        return {"rel": 2.5e-3}           # measured 6e-4
    if kind == "percall":
        return {"rel": 1.5e-5}           # measured 3e-6: populations as they are, not as offsets
    return {"rel": 4.0e-6}               # measured 7e-7


# ---- the same programs at 64 bits ----------------------------------------------------

_CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, -1, 1, 0, 0, -1, 1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1]
_CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1, 0, 0, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1]
_CZ = [0, 0, 0, 0, 0, -1, 1, 0, 0, 0, 0, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, -1, 1, -1, 1]


class _Lattice:
    def __init__(self, nl):
        self.c = torch.tensor([_CX[:nl], _CY[:nl], _CZ[:nl]], dtype=torch.float64, device="cuda").T.contiguous()
        tab = {19: (1 / 3, 1 / 18, 1 / 36, 0.0), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}[nl]
        self.w = torch.tensor([tab[int(s)] for s in (self.c ** 2).sum(1).tolist()], dtype=torch.float64, device="cuda")
        self.ci = [(_CX[l], _CY[l], _CZ[l]) for l in range(nl)]
        x, y, z = self.c.T
        self.cc = torch.stack([x * x, y * y, z * z, x * y, x * z, y * z], dim=1)      # (nl, 6)
        self.find = {c: l for l, c in enumerate(self.ci)}
        self.opp = [self.find[(-a, -b, -c)] for a, b, c in self.ci]


class _Exact:
    """The step of the reference on arrays f[l, k, j, i], ghost cells included."""

    def __init__(self, case, uvel, mask=None, turb=None):
        self.p, self.L = case, _Lattice(case["nl"])
        self.nx, self.ny, self.nz = case["nx"], case["ny"], case["nz"]
        self.uvel = uvel.double()
        self.mask = None if mask is None else (mask[1:-1, 1:-1, 1:-1] != 0)
        self.turb = None if turb is None else [t.double() for t in turb]
        self.eps = math.sqrt(2.2250738585072014e-308 if case["storage"] == "f64" else 1.17549435e-38)

    def feq(self, rho, u):
        """(nl, n) from rho (n), u (3, n)"""
        L = self.L
        cu, us = L.c @ u, (u * u).sum(0)
        return L.w[:, None] * rho * (1 + 3 * cu + 4.5 * cu ** 2 - 1.5 * us + 4.5 * cu * (cu ** 2 - us))

    def collide(self, f, rho, u):
        L = self.L
        fn = f - self.feq(rho, u)
        a = L.cc.T @ fn
        a = torch.cat([a[:3] - fn.sum(0) / 3, a[3:]])
        xx, yy, zz, xy, xz, yz = a
        mag = (xx ** 2 + yy ** 2 + zz ** 2 + 2 * (xy ** 2 + xz ** 2 + yz ** 2)).clamp_min(1.0e-300)
        e = self.eps
        b11, b22, b33 = e + xx * xx + xy * xy + xz * xz, e + xy * xy + yy * yy + yz * yz, e + xz * xz + yz * yz + zz * zz
        b12, b13, b23 = e + xx * xy + xy * yy + xz * yz, e + xx * xz + xy * yz + xz * zz, e + xy * xz + yy * yz + yz * zz
        t = (b11 * b22 - b12 ** 2 + b11 * b33 - b13 ** 2 + b22 * b33 - b23 ** 2) / mag
        on = t > e
        nut = torch.where(on, 2.5 * SMAG * SMAG * torch.sqrt(torch.where(on, t, torch.ones_like(t))), torch.zeros_like(t))
        K = 1 - 1 / (3 * (VISC + nut) + 0.5)
        cu = L.c @ u
        two = torch.tensor([1, 1, 1, 2, 2, 2], dtype=torch.float64, device="cuda")
        cac = (L.cc * two) @ a
        v = torch.stack([xx * u[0] + xy * u[1] + xz * u[2], xy * u[0] + yy * u[1] + yz * u[2],
                         xz * u[0] + yz * u[1] + zz * u[2]])
        tr = xx + yy + zz
        R = 4.5 * L.w[:, None] * (cac - tr / 3 + cu * (3 * cac - tr) - 2 * (L.c @ v))
        return self.feq(rho, u) + K * R

    def macro(self, f):
        rho = f.sum(0)
        return rho, torch.einsum("la,lkji->akji", self.L.c, f) / rho

    def postcoll(self, f, rho, u, it):
        """collision, turbulence slice and solid swap of the interior cells, in place"""
        inner = (slice(1, -1),) * 3
        step = max(1, 2_000_000 // (self.nx * self.ny)) if not torch.is_grad_enabled() else self.nz
        for k in range(1, self.nz + 1, step):
            s = (slice(k, min(k + step, self.nz + 1)), slice(1, -1), slice(1, -1))
            r = rho[s]
            f[(slice(None), *s)] = self.collide(f[(slice(None), *s)].reshape(self.L.w.numel(), -1), r.reshape(-1),
                                                u[(slice(None), *s)].reshape(3, -1)).reshape(-1, *r.shape)
        if self.turb is not None:
            i, lev = min(10, self.nx), it % LEVELS or LEVELS
            r, uu = rho[1:-1, 1:-1, i].reshape(-1), u[:, 1:-1, 1:-1, i].reshape(3, -1)
            du = AMPL * torch.stack([t[lev].reshape(-1) for t in self.turb])
            f[:, 1:-1, 1:-1, i] += (self.feq(r, uu + du) - self.feq(r, uu)).reshape(-1, self.nz, self.ny)
        if self.mask is not None:
            q = f[(slice(None), *inner)]
            f[(slice(None), *inner)] = torch.where(self.mask, q[self.L.opp], q)

    def periodic(self, f):
        p = self.p
        if p["ibnd"] == 0:
            f[..., 0], f[..., -1] = f[..., -2].clone(), f[..., 1].clone()
        f[:, :, 0], f[:, :, -1] = f[:, :, -2].clone(), f[:, :, 1].clone()
        if p["kbnd"] == 0:
            f[:, 0], f[:, -1] = f[:, -2].clone(), f[:, 1].clone()

    def boundary(self, f1, f2):
        """boundarycond: f1's ghost cells, in place"""
        L, nx, ny, nz = self.L, self.nx, self.ny, self.nz
        self.periodic(f1)
        if self.p["kbnd"]:
            lo, hi = {11: (-1, -1), 12: (-1, 1), 21: (1, -1), 22: (1, 1)}[self.p["kbnd"]]
            old = f1.clone()
            for side, opt in ((0, lo), (-1, hi)):
                kp = 1 if side == 0 else -2
                for l, (cx, cy, cz) in enumerate(L.ci):
                    if (cz >= 0) if side == 0 else (cz <= 0):
                        continue
                    f1[L.find[(opt * cx, opt * cy, -cz)], side, 1:-1, 1:-1] = f2[l, side, 1:-1, 1:-1]
                    f1[l, side, 1:-1, 1:-1] = old[l, kp, 1 - cy:ny + 1 - cy, 1 - cx:nx + 1 - cx]
        if self.p["ibnd"] == 1:
            fg = f1[:, 1:-1, 1:-1, 1] - 6 * (L.w * L.c[:, 0])[:, None, None] * self.uvel[None, :, None]
            f1[:, 1:-1, 1:-1, 0] = fg[[L.opp[l] if c[0] > 0 else l for l, c in enumerate(L.ci)]]
            f1[:, 1:-1, 1:-1, -1] = f1[:, 1:-1, 1:-1, -2].clone()
        self.periodic(f1)

    def drift(self, f2, f1):
        nx, ny, nz = self.nx, self.ny, self.nz
        for l, (cx, cy, cz) in enumerate(self.L.ci):
            f2[l, 1:-1, 1:-1, 1:-1] = f1[l, 1 - cz:nz + 1 - cz, 1 - cy:ny + 1 - cy, 1 - cx:nx + 1 - cx]

    def initial(self, macro):
        rho, u = macro[0].double(), torch.stack([m.double() for m in macro[1:]])
        fb = torch.zeros((self.L.w.numel(), *rho.shape), dtype=torch.float64, device="cuda")
        for k in range(1, self.nz + 1):
            r = rho[k, 1:-1, 1:-1]
            fb[:, k, 1:-1, 1:-1] = self.feq(r.reshape(-1), u[:, k, 1:-1, 1:-1].reshape(3, -1)).reshape(-1, *r.shape)
        for d in (1, 2, 3):                     # ghost cells copy the nearest interior cell
            fb.select(d, 0).copy_(fb.select(d, 1))
            fb.select(d, -1).copy_(fb.select(d, -2))
        fa = fb.clone()
        self.boundary(fb, fa)
        self.boundary(fa, fb)
        return fa, fb, rho, u

    def out(self, f1, f2):
        rho, u = self.macro(f1)
        return {"rho": rho, "u": u[0], "v": u[1], "w": u[2], "f1": f1.permute(1, 2, 3, 0), "f2": f2.permute(1, 2, 3, 0)}


def _run_exact(x, state, steps):
    f1, f2, rho, u = state
    for it in range(1, steps + 1):
        x.postcoll(f1, rho, u, it)
        x.boundary(f1, f2)
        x.drift(f2, f1)
        f1, f2 = f2, f1
        rho, u = x.macro(f1)
    return f1, f2


def _exact_slabs(case, d):
    n = case["tiles"]
    ny = case["ny"] // n
    tile = dict(case, ny=ny)
    whole = _Exact(case, d["uvel"])
    xs, st = [], []
    f1, f2, rho, u = whole.initial(d["macro"])
    for r in range(n):
        rows = slice(r * ny, (r + 1) * ny + 2)
        xs.append(_Exact(tile, d["uvel"], None if d["mask"] is None else d["mask"][:, rows]))
        st.append([f1[:, :, rows].clone(), f2[:, :, rows].clone(), rho[:, rows], u[:, :, rows]])
    for it in range(1, case["steps"] + 1):
        for x, s in zip(xs, st):
            x.postcoll(s[0], s[2], s[3], it)
            x.boundary(s[0], s[1])
        south, north = [s[0][:, :, 1].clone() for s in st], [s[0][:, :, -2].clone() for s in st]
        for r, (x, s) in enumerate(zip(xs, st)):
            s[0][:, :, 0], s[0][:, :, -1] = north[(r - 1) % n], south[(r + 1) % n]
            x.drift(s[1], s[0])
            s[0], s[1] = s[1], s[0]
            s[2], s[3] = x.macro(s[0])
    out = {}
    for r, (x, s) in enumerate(zip(xs, st)):
        out.update({"%s_%d" % kv: v for kv, v in zip(((k, r) for k in ("rho", "u", "v", "w", "f1", "f2")), x.out(*s[:2]).values())})
    return out


def _exact_gradient(case, d):
    x = _Exact(case, d["uvel"], d["mask"])
    f1 = d["f1"].double().permute(3, 0, 1, 2).contiguous().requires_grad_()
    uvel = d["uvel"].double().requires_grad_()
    f2 = d["f2"].double().permute(3, 0, 1, 2).contiguous()

    def step(a, b, uv):
        x.uvel = uv
        a, b = a.clone(), b.clone()
        rho, u = x.macro(a)
        x.postcoll(a, rho, u, 0)
        x.boundary(a, b)
        x.drift(b, a)
        return b, a

    with torch.enable_grad():
        a, b = f1, f2
        for _ in range(case["steps"]):
            a, b = checkpoint(step, a, b, uvel, use_reentrant=False)
        pr = torch.from_numpy(d["probes"]).cuda()
        at = a[:, pr[:, 2], pr[:, 1], pr[:, 0]]
        u = (at.T @ x.L.c) / at.sum(0)[:, None]
        loss = 0.5 * ((u - d["target"].double()) ** 2).sum()
        g, gu = torch.autograd.grad(loss, (f1, uvel))
    return {"u": u.detach(), "f1_grad": g.permute(1, 2, 3, 0), "uvel_grad": gu}


def _exact_turbulence(case, seed):
    """Gaussian amplitudes with hashed phases, one inverse transform per level, then
    the levels chained and normalised in order."""
    ny, nz, nt = case["ny"], case["nz"], case["nrturb"] + 1
    n1, n2 = ny + ny % 2, nz + nz % 2
    h, s2 = n1 // 2 + 1, 8.0 * 3.0 / 100.0
    k2, l2 = (2 * math.pi / n1) ** 2, (2 * math.pi / n2) ** 2
    pp, ll = np.meshgrid(np.arange(-n2 // 2 + 1, n2 // 2 + 1), np.arange(-n1 // 2 + 1, n1 // 2 + 1), indexing="ij")
    amp = 1.0 / math.sqrt(np.exp(-2.0 * (k2 * ll ** 2 + l2 * pp ** 2) / s2).sum() - 1.0)

    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    p = np.arange(n2)
    p = np.where(p < n2 // 2, p, p - n2)[:, None] + np.zeros((1, h), np.int64)
    l = np.arange(h)[None, :] + np.zeros((n2, 1), np.int64)
    edge = (l == 0) | (l == n1 // 2)
    flip = edge & (p < 0) & (p != -(n2 // 2))
    p = np.where(flip, -p, p)
    mod = amp * np.exp(-(k2 * l ** 2 + l2 * p ** 2) / s2)
    real = edge & ((p == 0) | (p == -(n2 // 2)))
    mod[(l == 0) & (p == 0)] = 0.0
    base = ((p + n2 // 2) * h + l).astype(np.uint64)
    mod, real, flip = (torch.from_numpy(a).cuda() for a in (mod, real, flip))
    out = []
    with np.errstate(over="ignore"):
        for f in range(case["fields"]):
            lev = torch.empty((nt, nz, ny), dtype=torch.float64, device="cuda")
            for t in range(nt):
                b = f * nt + t
                bits = mix(np.uint64(seed) ^ mix(base + np.uint64(b * (n2 + 1) * h))) >> np.uint64(40)
                phi = torch.from_numpy(bits.astype(np.float64)).cuda() * (2 * math.pi / 16777216.0)
                im = torch.where(real, torch.zeros_like(phi), torch.where(flip, -1.0, 1.0) * mod * torch.sin(phi))
                y = torch.fft.irfft2(torch.complex(mod * torch.cos(phi), im), s=(n2, n1), norm="forward")[:nz, :ny]
                if t:
                    y = 0.98 * lev[t - 1] + math.sqrt(1 - 0.98 ** 2) * y
                    y = y - y.mean()
                    y = y / torch.sqrt((y * y).sum() / (ny * nz - 1))
                lev[t] = y
            out.append(lev)
    return out


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "turbulence":
            return _exact_turbulence(case, int(seed))
        if kind == "ensemble":
            got = []
            for m in _members(case, seed):
                d = _member_inputs(m)
                x = _Exact(m, d["uvel"], turb=d["turb"])
                f1, _ = _run_exact(x, x.initial(d["macro"]), m["steps"])
                rho, u = x.macro(f1)
                got.append([t.reshape(-1) for t in (rho, *u)])
            return {n: torch.cat([g[q] for g in got]) for q, n in enumerate(("rho", "u", "v", "w"))}
        if kind.startswith("adjoint"):
            return _exact_gradient(case, _probe_inputs(case, seed))
        d = _inputs(case, seed)
        if kind == "slabs":
            return _exact_slabs(case, d)
        x = _Exact(case, d["uvel"], d["mask"], d["turb"])
        return x.out(*_run_exact(x, x.initial(d["macro"]), case["steps"]))
