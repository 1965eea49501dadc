"""The steady step at the edges of its launch shapes: rows that end inside a block of
any width, odd row lengths (a last pair with one cell), and periodic boxes; against the
one-cell kernel and the per-call path."""
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
