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
