"""External forcing (forcings_apply): per call and fused into the step, against the oracle."""
import numpy as np
import pytest

from lbm_b200 import workloads as W
from oracle import oracle as O
from tests.test_gpu_fused import SMALL, compare_to_floor, cuda, host, params_of, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl", [19, 27])
def test_forcings_apply_per_call(nl):
    from lbm_b200 import Lbm, Params
    cfg = O.Config(13, 7, 6, nl)
    rng = np.random.default_rng(5)
    f = rng.uniform(0.0, 0.1, cfg.fshape).astype(np.float32)
    rho = (1.0 + 0.01 * rng.standard_normal(cfg.sshape)).astype(np.float32)
    u, v, w = ((0.03 * rng.standard_normal(cfg.sshape)).astype(np.float32) for _ in range(3))
    F = (1e-4 * rng.standard_normal(cfg.sshape + (3,))).astype(np.float32)
    refs = {}
    for dt in (np.float32, np.float64):
        g = f.astype(dt)
        O.Oracle(cfg, dt).forcings_apply(g, F.astype(dt), *(a.astype(dt) for a in (rho, u, v, w)))
        refs[dt] = g
    L = Lbm(Params(nx=13, ny=7, nz=6, nl=nl, iturb_pos=3))
    fg = cuda(f)
    L.forcings_apply(fg, cuda(F), *(cuda(a) for a in (rho, u, v, w)))
    out = host(fg).astype(np.float64)
    # the reference forms feq1 - feq0 as a difference of two O(0.05) values; the closed form
    # used here is closer to FP64, so the bound is the FP32 oracle's own distance to FP64
    floor = np.abs(refs[np.float32] - refs[np.float64]).max()
    e64 = np.abs(out - refs[np.float64]).max()
    e32 = np.abs(out - refs[np.float32]).max()
    assert e64 <= 1.5 * floor + 1e-9 and e32 <= 2.5 * floor + 1e-9, (e64, e32, floor)


def run_forced(wl, steps, storage, F, kernel=None, slice_on=True):
    from lbm_b200 import Solver
    blank = W.blanking(wl)
    rho, u, v, w = (cuda(a) for a in W.initial_macro(wl))
    uvel = cuda(W.inflow_profile(wl))
    turb = W.turbulence_fields(wl.ny, wl.nz, wl.nrturb, 3)
    tb = (cuda(turb[0]), cuda(turb[1]), cuda(turb[2]), wl.nrturb, wl.ampl) if slice_on else None
    s = Solver(params_of(wl, iturb_pos=5, storage=storage), rho, u, v, w, uvel, blanking=cuda(blank), turbulence=tb)
    if kernel:
        s.lbm.set_kernel(kernel)
    Fg = cuda(F)
    s.lbm.set_forcing(Fg)
    s.step(steps)
    f1, f2 = s.state()
    r, uu, vv, ww = s.macro()
    out = tuple(host(t) for t in (f1, f2, r, uu, vv, ww))
    s.close()
    return out


def oracle_forced(wl, steps, dtype, F, slice_on=True):
    blank = W.blanking(wl)
    turb = W.turbulence_fields(wl.ny, wl.nz, wl.nrturb, 3)
    cfg = O.Config(wl.nx, wl.ny, wl.nz, wl.nl, ibnd=wl.ibnd, jbnd=wl.jbnd, kbnd=wl.kbnd, iturb_pos=5, lsolids=True,
                   lturb=slice_on, nrturb=wl.nrturb, kinevisc=wl.kinevisc, ampl=wl.ampl)
    o = O.Oracle(cfg, dtype)
    rho, u, v, w = (a.astype(dtype) for a in W.initial_macro(wl))
    uvel = W.inflow_profile(wl, dtype)
    fA, fB = o.zeros_f(), o.zeros_f()
    o.init(fA, fB, rho, u, v, w, uvel)
    tau = np.full(cfg.sshape, 3 * np.float32(wl.kinevisc) + 0.5, dtype)
    o.run(fA, fB, rho, u, v, w, tau, uvel, steps, blanking=blank, uu=turb[0].astype(dtype),
          vv=turb[1].astype(dtype), ww=turb[2].astype(dtype), force=F.astype(dtype))
    return fA, fB, rho, u, v, w


@pytest.mark.parametrize("nl", [19, 27])
def test_fused_forcing_matches_oracle(nl):
    wl = SMALL.with_(nl=nl)
    F = (2e-5 * np.random.default_rng(9).standard_normal((wl.nz + 2, wl.ny + 2, wl.nx + 2, 3))).astype(np.float32)
    gpu = run_forced(wl, wl.steps, "f32", F)
    ref32, ref64 = oracle_forced(wl, wl.steps, np.float32, F), oracle_forced(wl, wl.steps, np.float64, F)
    compare_to_floor(gpu, ref32, ref64, "forced")
    # the forcing does something: without it the run differs well beyond the floor
    unforced = run_forced(wl, wl.steps, "f32", np.zeros_like(F))
    assert rel_l2(unforced[3], ref64[3]) > 100 * rel_l2(gpu[3], ref64[3])


@pytest.mark.parametrize("codes", [(0, 0, 0), (11, 0, 22), (12, 0, 0), (1, 11, 22)])
@pytest.mark.parametrize("nl,storage,nx", [(19, "f32", 16), (27, "f32", 34), (27, "f16", 34), (27, "f16", 512)])
def test_fused_forcing_outside_the_folded_configuration(codes, nl, storage, nx):
    """Periodic boxes, where the forced kernel writes the i ghosts, and boxes with closed faces,
    where an instance without those stores runs; FP16 D3Q27 in both widths of block."""
    ib, jb, kb = codes
    wl = SMALL.with_(nl=nl, nx=nx, ny=6, nz=5, ibnd=ib, jbnd=jb, kbnd=kb)
    F = (2e-5 * np.random.default_rng(9).standard_normal((wl.nz + 2, wl.ny + 2, wl.nx + 2, 3))).astype(np.float32)
    gpu = run_forced(wl, 10, storage, F, slice_on=False)
    ref32, ref64 = (oracle_forced(wl, 10, dt, F, slice_on=False) for dt in (np.float32, np.float64))
    if storage == "f32":
        compare_to_floor(gpu, ref32, ref64, "forced, codes %s" % (codes,))
    else:
        s = (slice(1, -1),) * 3
        assert rel_l2(np.stack(gpu[3:])[(slice(None),) + s], np.stack(ref64[3:])[(slice(None),) + s]) < 1e-3


def test_fused_forcing_fp16_storage():
    wl = SMALL
    F = (2e-5 * np.random.default_rng(9).standard_normal((wl.nz + 2, wl.ny + 2, wl.nx + 2, 3))).astype(np.float32)
    g16 = run_forced(wl, 40, "f16", F)
    ref64 = oracle_forced(wl, 40, np.float64, F)
    s = (slice(1, -1),) * 3
    assert rel_l2(np.stack(g16[3:])[(slice(None),) + s], np.stack(ref64[3:])[(slice(None),) + s]) < 1e-3


def test_fused_forcing_needs_the_pair_kernel():
    from lbm_b200 import LbmError
    wl = SMALL.with_(steps=2)
    F = np.zeros((wl.nz + 2, wl.ny + 2, wl.nx + 2, 3), np.float32)
    with pytest.raises(LbmError, match="two-cells-per-thread"):
        run_forced(wl, 3, "f32", F, kernel="pull")
