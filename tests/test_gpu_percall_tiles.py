"""The per-call kernels at the edges of their tiles: rows shorter than a chunk, one
cell past it, rows and planes that do not fill a tile, and arrays at every
alignment an element type allows."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

C = torch.tensor([[0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, -1, 1, 0, 0, -1, 1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1],
                  [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1, 0, 0, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1],
                  [0, 0, 0, 0, 0, -1, 1, 0, 0, 0, 0, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, -1, 1, -1, 1]]).T.tolist()
SHAPES = [(2, 2, 2), (5, 3, 2), (31, 4, 3), (32, 5, 9), (33, 8, 6), (64, 3, 5), (101, 9, 4), (130, 6, 7)]


def lbm_of(nx, ny, nz, nl, **kw):
    from lbm_b200 import Lbm, Params
    return Lbm(Params(nx=nx, ny=ny, nz=nz, nl=nl, iturb_pos=2, **kw))


def at_offset(shape, dtype, off, g):
    """a random array whose first element sits `off` elements past an aligned address"""
    n = 1
    for s in shape:
        n *= s
    base = torch.randn(n + 8, dtype=dtype, device="cuda", generator=g)
    return base[off:off + n].view(shape)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", SHAPES)
def test_drift_moves_every_value(shape, nl, dtype):
    nx, ny, nz = shape
    L = lbm_of(nx, ny, nz, nl)
    g = torch.Generator(device="cuda")
    g.manual_seed(nx * 100 + ny)
    for fo, so in ((0, 0), (1, 3), (2, 1), (3, 2)):
        f = at_offset(L.p.fshape, dtype, fo, g)
        src = at_offset(L.p.fshape, dtype, so, g)
        want, keep = f.clone(), src.clone()
        for l in range(nl):
            cx, cy, cz = C[l]
            want[1:-1, 1:-1, 1:-1, l] = src[1 - cz:nz + 1 - cz, 1 - cy:ny + 1 - cy, 1 - cx:nx + 1 - cx, l]
        L.drift(f, src)
        assert torch.equal(f, want) and torch.equal(src, keep)     # ghosts and the source stay as they were
    L.close()


def equilibrium_like(nl, shape, dtype, off, g):
    """rho, u, v, w and an f near their equilibrium, at an alignment offset"""
    sc = [torch.randn(shape, dtype=dtype, device="cuda", generator=g) * 0.02 for _ in range(4)]
    sc[0] += 1.0
    sc[1] += 0.05
    f = at_offset(shape + (nl,), dtype, off, g)
    w = torch.tensor([{19: (1 / 3, 1 / 18, 1 / 36, 0), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}[nl][sum(x * x for x in c)]
                      for c in C[:nl]], dtype=dtype, device="cuda")
    f.mul_(0.02).add_(1.0).mul_(w)
    return f, sc


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", SHAPES)
def test_postcoll_and_macrovars(shape, nl, dtype):
    import numpy as np

    from oracle import oracle as O
    nx, ny, nz = shape
    L = lbm_of(nx, ny, nz, nl)
    o = O.Oracle(O.Config(nx, ny, nz, nl, iturb_pos=2), np.float64)
    g = torch.Generator(device="cuda")
    g.manual_seed(nx * 100 + nz)
    s = (slice(1, -1),) * 3
    for off in range(16 // dtype.itemsize):
        f, sc = equilibrium_like(nl, L.p.sshape, dtype, off, g)
        tau = torch.full(L.p.sshape, 0.5, dtype=dtype, device="cuda")
        # macrovars: every cell, in the order of the directions, bit for bit
        want = [torch.zeros_like(sc[0]) for _ in range(4)]
        for l in range(nl):
            want[0] += f[..., l]
            for a in range(3):
                want[a + 1] += C[l][a] * f[..., l]
        inv = 1.0 / want[0]
        out = [torch.full_like(sc[0], 9.0) for _ in range(4)]
        L.macrovars(*out, f)
        assert torch.equal(out[0], want[0]) and all(torch.equal(out[a], want[a] * inv) for a in (1, 2, 3))
        # postcoll: the interior against the FP64 oracle, the ghosts and their tau untouched
        before = f.clone()
        rf, rt = (t.double().cpu().numpy().copy() for t in (f, tau))
        o.postcoll(rf, rt, *(t.double().cpu().numpy() for t in sc))
        L.postcoll(f, tau, *sc)
        got, gt = f.double().cpu().numpy(), tau.double().cpu().numpy()
        tol = 2e-6 if dtype == torch.float32 else 1e-13       # as test_gpu_percall.py: closed form against dense loops
        assert np.linalg.norm(got[s] - rf[s]) < tol * np.linalg.norm(rf[s])
        assert np.linalg.norm(gt[s] - rt[s]) < 100 * tol * np.linalg.norm(rt[s] - 0.5) + 1e-7 * (dtype == torch.float32) * rt[s].size ** 0.5
        f[s] = before[s]
        assert torch.equal(f, before)
        tau[s] = 0.5
        assert bool((tau == 0.5).all())
    L.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 2), (33, 8, 6), (64, 3, 5)])
def test_boundarycond_of_every_kind(shape, nl, dtype):
    """Copies bit for bit against the oracle, for periodic, closed and inflow axes in
    combination (the j copies a face reads through, the edges and the corners)."""
    import numpy as np

    from oracle import oracle as O
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + ny)
    real = np.float32 if dtype == torch.float32 else np.float64
    for ib, jb, kb in ((1, 0, 12), (1, 0, 0), (0, 0, 0), (0, 0, 12), (0, 0, 21), (11, 0, 22), (11, 0, 0), (0, 11, 12), (1, 12, 11),
                       (22, 22, 22), (12, 21, 0)):
        L = lbm_of(nx, ny, nz, nl, ibnd=ib, jbnd=jb, kbnd=kb, udir=10.0)
        o = O.Oracle(O.Config(nx, ny, nz, nl, ibnd=ib, jbnd=jb, kbnd=kb, iturb_pos=2, udir=10.0), real)
        a, b = (rng.standard_normal(L.p.fshape).astype(real) for _ in range(2))
        uvel = rng.standard_normal(nz).astype(real)
        da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        L.boundarycond(da, db, torch.from_numpy(uvel).cuda())
        o.boundarycond(a, b, uvel)
        got = da.cpu().numpy()
        assert np.array_equal(db.cpu().numpy(), b)
        if ib == 1:
            # the inflow value: a product and a difference, rounded once or twice
            assert np.abs(got - a).max() < 8 * np.finfo(real).eps * max(1.0, np.abs(a).max()), (ib, jb, kb)
            assert np.array_equal(got[:, :, 1:], a[:, :, 1:])
        else:
            assert np.array_equal(got, a), (ib, jb, kb)
        L.close()


@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 2), (33, 8, 6), (130, 6, 7)])
def test_solids_at_every_mask_alignment(shape, nl):
    nx, ny, nz = shape
    L = lbm_of(nx, ny, nz, nl)
    g = torch.Generator(device="cuda")
    g.manual_seed(nx)
    n = (nx + 2) * (ny + 2) * (nz + 2)
    swap = [0] + [l + 1 if l % 2 else l - 1 for l in range(1, nl)]
    for off in range(4):
        base = (torch.rand(n + 8, device="cuda", generator=g) < 0.3).to(torch.int32) * -1     # a Fortran .true. is any nonzero
        blank = base[off:off + n].view(L.p.sshape)
        f = at_offset(L.p.fshape, torch.float32, off, g)
        want = f.clone()
        s = (slice(1, -1),) * 3
        want[s] = torch.where(blank[s][..., None] != 0, f[s][..., swap], f[s])
        L.solids(f, blank)
        assert torch.equal(f, want)
    L.close()
