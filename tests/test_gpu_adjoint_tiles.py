"""The adjoint kernels at the edges of their tiles: the drift transpose against its
definition, the boundary transpose against its forward (a linear map), and the collision
adjoint of a row against the same cells elsewhere in a row."""
import pytest

from tests.test_gpu_percall_tiles import C, SHAPES, at_offset, equilibrium_like, lbm_of

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", SHAPES)
def test_drift_transpose(shape, nl):
    nx, ny, nz = shape
    L = lbm_of(nx, ny, nz, nl)
    g = gen(nx * 10 + nz)
    s = (slice(1, -1),) * 3
    for io, oo in ((0, 0), (1, 2), (3, 1)):
        fin = at_offset(L.p.fshape, torch.float32, io, g)
        fout = at_offset(L.p.fshape, torch.float32, oo, g)
        want = fin.clone()
        for l in range(nl):
            cx, cy, cz = C[l]
            want[1 - cz:nz + 1 - cz, 1 - cy:ny + 1 - cy, 1 - cx:nx + 1 - cx, l] += fout[s + (l,)]
        cleared = fout.clone()
        cleared[s] = 0.0
        a, b = fin.clone(), fout.clone()
        L.drift_adj(fin, fout)
        assert torch.equal(fin, want) and torch.equal(fout, cleared)
        # with the macrovars adjoint in front
        sc = [torch.randn(L.p.sshape, device="cuda", generator=g) for _ in range(7)]
        rho = 1.0 + 0.1 * torch.rand(L.p.sshape, device="cuda", generator=g)
        rh, uh, vh, wh, u, v, w = sc
        t = [rh - (uh * u + vh * v + wh * w) / rho] + [x / rho for x in (uh, vh, wh)]
        want = a.double()
        for l in range(nl):
            cx, cy, cz = C[l]
            m = t[0] + cx * t[1] + cy * t[2] + cz * t[3]
            want[1 - cz:nz + 1 - cz, 1 - cy:ny + 1 - cy, 1 - cx:nx + 1 - cx, l] += (b[..., l] + m)[s]
        L.macrovars_drift_adj(a, b, rh, uh, vh, wh, rho, u, v, w)
        # sums of about ten values below 10, each rounded to 6e-8
        assert float((a - want).abs().max()) < 1e-5 and torch.equal(b, cleared)
    L.close()


@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 2), (33, 8, 6)])
def test_boundary_transpose(shape, nl):
    """<y, B x> = <B^T y, x> for the linear map (f1, f2, uvel) -> (f1, f2) of boundarycond."""
    nx, ny, nz = shape
    g = gen(nx)
    for ib, jb, kb in ((1, 0, 12), (1, 0, 0), (0, 0, 0), (0, 0, 21), (11, 0, 22), (11, 0, 0), (0, 11, 12), (1, 12, 11), (22, 22, 22)):
        L = lbm_of(nx, ny, nz, nl, ibnd=ib, jbnd=jb, kbnd=kb, udir=10.0)
        x = [torch.randn(L.p.fshape, device="cuda", generator=g) for _ in range(2)]
        y = [torch.randn(L.p.fshape, device="cuda", generator=g) for _ in range(2)]
        uv = torch.randn(nz, device="cuda", generator=g)
        bx = [t.clone() for t in x]
        L.boundarycond(bx[0], bx[1], uv)
        ty = [t.clone() for t in y]
        tu = torch.zeros(nz, device="cuda")
        L.boundarycond_adj(ty[0], ty[1], tu)
        lhs = sum(float((p.double() * q.double()).sum()) for p, q in zip(y, bx))
        rhs = sum(float((p.double() * q.double()).sum()) for p, q in zip(ty, x)) + float((tu.double() * uv.double()).sum())
        n = x[0].numel() ** 0.5
        assert abs(lhs - rhs) < 2e-6 * n * 4, (ib, jb, kb, lhs, rhs)      # sums of n^2 terms of order one, FP32 rounding each
        L.close()


@pytest.mark.parametrize("nl", [19, 27])
@pytest.mark.parametrize("shape", SHAPES)
def test_collision_adjoint_does_not_depend_on_the_place(shape, nl):
    """Each cell of a domain against the same cell in a domain of one row of two cells."""
    nx, ny, nz = shape
    L = lbm_of(nx, ny, nz, nl)
    n = nx * ny * nz
    S = lbm_of(n, 2, 2, nl)
    s = (slice(1, -1),) * 3
    g = gen(nx + nz)
    for off in range(4):
        f, sc = equilibrium_like(nl, L.p.sshape, torch.float32, off, g)
        fh = at_offset(L.p.fshape, torch.float32, (off + 1) % 4, g)
        hats = [torch.randn(L.p.sshape, device="cuda", generator=g) for _ in range(4)]
        blank = (torch.rand(L.p.sshape, device="cuda", generator=g) < 0.2).to(torch.int32)
        before, hbefore = fh.clone(), [h.clone() for h in hats]

        def row(a):
            b = torch.ones(S.p.sshape + a.shape[3:], dtype=a.dtype, device="cuda")
            b[1, 1, 1:-1] = a[s].reshape((n,) + a.shape[3:])
            return b
        want, hw = row(fh), [row(h) for h in hats]
        S.postcoll_adj(want, row(f), *(row(t) for t in sc), *hw, blanking=row(blank))
        L.postcoll_adj(fh, f, *sc, *hats, blanking=blank)
        assert torch.equal(fh[s].reshape(n, nl), want[1, 1, 1:-1])
        assert all(torch.equal(h[s].reshape(n), q[1, 1, 1:-1]) for h, q in zip(hats, hw))
        fh[s] = before[s]
        assert torch.equal(fh, before)
        for h, q in zip(hats, hbefore):
            h[s] = q[s]
            assert torch.equal(h, q)
    L.close()
    S.close()
