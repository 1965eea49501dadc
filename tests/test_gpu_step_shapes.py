"""The steady step at the edges of its launch shapes: rows that end inside a block of
any width, odd row lengths (a last pair with one cell), and periodic boxes; against the
one-cell kernel, the per-call path and a step at 64 bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def make(nx, ny, nz, nl, storage, codes, solids, turb, fused=True, kernel=None):
    from lbm_b200 import Params, Solver
    g = torch.Generator(device="cuda")
    g.manual_seed(nx * 7 + ny)
    ib, jb, kb = codes
    p = Params(nx=nx, ny=ny, nz=nz, nl=nl, ibnd=ib, jbnd=jb, kbnd=kb, iturb_pos=min(nx, 3), storage=storage)
    m = [torch.zeros(p.sshape, device="cuda") for _ in range(4)]
    s = (slice(1, -1),) * 3
    m[0][s] = 1.0
    for q in (1, 2, 3):
        m[q][s] = 0.02 * torch.randn((nz, ny, nx), device="cuda", generator=g) + (0.05 if q == 1 else 0.0)
    mask = None
    if solids:
        mask = torch.zeros(p.sshape, dtype=torch.int32, device="cuda")
        mask[s] = (torch.rand((nz, ny, nx), device="cuda", generator=g) < 0.1).to(torch.int32)
    t = None
    if turb:
        t = (*(torch.randn((4, nz, ny), device="cuda", generator=g) for _ in range(3)), 3, 1e-3)
    sol = Solver(p, *m, torch.full((nz,), 0.05, device="cuda"), blanking=mask, turbulence=t, fused=fused)
    if kernel:
        sol.lbm.set_kernel(kernel)
    return sol


def agree(a, b, tol):
    for x, y in zip(a.state() + a.macro(), b.state() + b.macro()):
        assert bool(torch.isfinite(x).all())
        assert float((x - y).abs().max()) < tol, float((x - y).abs().max())


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("nx", [4, 5, 7, 63, 64, 65, 66, 127, 128, 129, 191, 192, 255, 257, 512])
def test_pair_kernel_against_one_cell_kernel(nx, nl, storage):
    # FP32: rounding of populations below 0.3 over five steps; FP16: a step of the offset grid,
    # 2^-11 of 2e-2, carried through them
    tol = 2e-6 if storage == "f32" else 2e-4
    for codes, solids, turb in (((1, 0, 12), True, True), ((1, 0, 21), False, True), ((0, 0, 0), True, False), ((0, 12, 11), True, False)):
        a = make(nx, 5, 4, nl, storage, codes, solids, turb)
        b = make(nx, 5, 4, nl, storage, codes, solids, turb, kernel="pull")
        for s in (a, b):
            s.step(5)
            assert s.lbm.status() == 0
        agree(a, b, tol)


@pytest.mark.parametrize("nx,ny,nz", [(4, 2, 2), (5, 3, 2), (33, 2, 7), (64, 5, 3), (130, 4, 4)])
@pytest.mark.parametrize("nl", [19, 27])
def test_periodic_box_against_percall(nx, ny, nz, nl):
    a = make(nx, ny, nz, nl, "f32", (0, 0, 0), True, False)
    b = make(nx, ny, nz, nl, "f32", (0, 0, 0), True, False, fused=False)
    for n in (1, 1, 3):
        a.step(n)
        b.step(n)
        agree(a, b, 2e-6)
        assert a.lbm.it == a.it


@pytest.mark.parametrize("codes,why", [((1, 0, 12), "forcing"), ((0, 0, 0), "forcing"), ((1, 0, 12), "slab")])
def test_odd_rows_refuse_what_they_did(codes, why):
    """External forcing and folded j slabs take an even nx, as before."""
    from lbm_b200 import LbmError
    s = make(9, 4, 4, 19, "f32", codes, False, False)
    if why == "forcing":
        s.lbm.set_forcing(torch.zeros(s.p.sshape + (3,), device="cuda"))
        with pytest.raises(LbmError):
            s.step(2)
    else:
        from lbm_b200 import Lbm
        L = Lbm(s.p)
        L.set_halo_j(True)
        f1, f2 = s.state()
        L.state_import(f1, f2, *s.macro())
        L.set_inflow(s.uvel)
        L.step(1)                     # collides in place
        with pytest.raises(LbmError):
            L.step(1)


def raw_state(sol):
    """(nl, nz, ny, nx) stored values of the newest buffer, interior cells."""
    p, L = sol.p, sol.lbm
    b = L.state_scratch()
    L.state_copy(b)
    pitch = (p.nx + 34 + 31) // 32 * 32
    rows = (p.ny + 2) * (p.nz + 2) * pitch
    v = b.view(torch.float16) if p.storage == "f16" else b
    v = v[:p.nl * (rows + 32)].view(p.nl, rows + 32)[:, :rows].view(p.nl, p.nz + 2, p.ny + 2, pitch)
    return v[:, 1:-1, 1:-1, 32:32 + p.nx].clone()


def step64(h, p, solid, scale):
    """The stored values after one step of a periodic box, at 64 bits (regularized third-order
    Hermite collision with the Vreman viscosity, bounce-back at solid cells)."""
    from oracle import oracle as O
    tab = O.tables(p.nl, np.float64)
    c = [[int(x) for x in tab[k]] for k in ("cx", "cy", "cz")]
    w = [float(x) for x in tab["w"]]
    Q = p.nl
    o = [torch.roll(h[l].double() / scale, (c[2][l], c[1][l], c[0][l]), (0, 1, 2)) for l in range(Q)]

    def moment(k):
        return sum(k(l) * o[l] for l in range(Q) if k(l))
    s0 = sum(o)
    rho = 1 + s0
    u = [moment(lambda l, a=a: c[a][l]) / rho for a in range(3)]
    A = [[moment(lambda l: c[a][l] * c[b][l]) - (s0 / 3 if a == b else 0) - rho * u[a] * u[b] for b in range(3)]
         for a in range(3)]
    tr = A[0][0] + A[1][1] + A[2][2]
    tiny = float(np.finfo(np.float32).tiny)
    eps = float(np.sqrt(np.float32(tiny)))
    sq = sum(A[a][b] ** 2 for a in range(3) for b in range(3))
    B = [[eps + sum(A[a][d] * A[b][d] for d in range(3)) for b in range(3)] for a in range(3)]
    t = sum(B[a][a] * B[b][b] - B[a][b] ** 2 for a, b in ((0, 1), (0, 2), (1, 2))) / sq.clamp(min=tiny)
    nut = torch.where(t > eps, 2.5 * p.smagorinsky ** 2 * t.clamp(min=0).sqrt(), torch.zeros_like(t))
    K = 1 - 1 / (3 * (p.kinevisc + nut) + 0.5)
    usq = sum(x * x for x in u)
    out = []
    for l in range(Q):
        cu = sum(c[a][l] * u[a] for a in range(3))
        cac = sum(c[a][l] * c[b][l] * A[a][b] for a in range(3) for b in range(3))
        cau = sum(c[a][l] * A[a][b] * u[b] for a in range(3) for b in range(3))
        out.append(w[l] * (s0 - 1.5 * rho * usq - 1.5 * K * tr + 4.5 * K * cac + 4.5 * rho * cu ** 2 - 9 * K * cau
                           + cu * (3 * rho - 4.5 * rho * usq - 4.5 * K * tr + 13.5 * K * cac + 4.5 * rho * cu ** 2)))
    swap = [out[0]] + [out[l + 1 if l % 2 else l - 1] for l in range(1, Q)]
    return torch.where(solid, torch.stack(swap), torch.stack(out)) * scale


@pytest.mark.parametrize("nl,storage,bound", [(19, "f32", 1.02), (27, "f32", 1.02), (19, "f16", 1.04), (27, "f16", 1.20)])
def test_odd_rows_round_as_the_one_cell_kernel(nl, storage, bound):
    """One step of an odd-nx box against 64 bits: the pair kernel's error is the one-cell
    kernel's.  FP32: the 2-norm (it was 1.045 of it with products rounded before they were
    summed).  FP16, where storage rounding hides the arithmetic: the share of stored values
    that are not the nearest to the exact one (D3Q19 1.08 of it with approximate reciprocals and
    unfused products, 1.00 now; D3Q27 1.13 by its separable emission).  3.5e7 values or more
    make the share good to 1%, the norm far better."""
    from lbm_b200 import Params, Solver
    p = Params(nx=101, ny=96, nz=96, nl=nl, ibnd=0, jbnd=0, kbnd=0, storage=storage, kinevisc=1e-4, smagorinsky=0.15)
    scale = 256.0 if storage == "f16" else 1.0
    it, ft = (torch.int16, torch.float16) if storage == "f16" else (torch.int32, torch.float32)
    inner = (slice(1, -1),) * 3
    err = {"pull": 0.0, "pair": 0.0}
    for seed in (1, 2):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        m = [torch.zeros(p.sshape, device="cuda") for _ in range(4)]
        m[0][inner] = 1.0 + 0.01 * torch.randn((p.nz, p.ny, p.nx), device="cuda", generator=g)
        for q in (1, 2, 3):
            m[q][inner] = 0.03 * torch.randn((p.nz, p.ny, p.nx), device="cuda", generator=g) + (0.05 if q == 1 else 0.0)
        mask = torch.zeros(p.sshape, dtype=torch.int32, device="cuda")
        mask[inner] = (torch.rand((p.nz, p.ny, p.nx), device="cuda", generator=g) < 0.05).to(torch.int32)
        for kernel in err:
            s = Solver(p, *m, torch.full((p.nz,), 0.05, device="cuda"), blanking=mask)
            s.lbm.set_kernel("pull")
            s.step(3)
            before = raw_state(s)
            s.lbm.set_kernel(kernel)
            s.step(1)
            got = raw_state(s)
            s.close()
            exact = step64(before, p, mask[inner] != 0, scale)
            d = (got.double() - exact).abs()
            if storage == "f16":
                near = [(got.view(it) + q).view(ft).double() for q in (1, -1)]
                err[kernel] += float(((near[0] - exact).abs() < d).logical_or((near[1] - exact).abs() < d).sum())
            else:
                err[kernel] += float(d.square().sum())
    ratio = err["pair"] / err["pull"] if storage == "f16" else (err["pair"] / err["pull"]) ** 0.5
    assert ratio < bound, ratio
