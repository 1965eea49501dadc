"""The fused gradient over every way its steps fall into segments: a single one, full and
short last ones, one step each; with and without overlap, twice in a row, and from a
forward run that kept another run's arrays before.  What a problem holds after it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsteps,K", [(1, 1), (2, 1), (5, 1), (3, 10), (4, 4), (8, 4), (9, 4), (11, 4), (13, 3)])
def test_segments_give_the_percall_gradient(nsteps, K, nx=20):
    from lbm_b200 import Lbm, Params
    from lbm_b200.adjoint import FusedProbeProblem, ProbeProblem, initial_state
    p = Params(nx=nx, ny=6, nz=8, nl=19, iturb_pos=2)
    g = torch.Generator(device="cuda")
    g.manual_seed(nsteps * 16 + K)
    m = [torch.zeros(p.sshape, device="cuda") for _ in range(4)]
    m[0][1:-1, 1:-1, 1:-1] = 1.0
    for q in (1, 2, 3):
        m[q][1:-1, 1:-1, 1:-1] = 0.03 * torch.randn((p.nz, p.ny, p.nx), device="cuda", generator=g)
    uvel = torch.full((p.nz,), 0.05, device="cuda")
    with Lbm(p) as L:
        f1, f2 = initial_state(L, *m, uvel)
        torch.cuda.synchronize()
    f1 *= 1.0 + 5e-3 * torch.randn(f1.shape, device="cuda", generator=g)      # away from exact equilibrium
    mask = torch.zeros(p.sshape, dtype=torch.int32, device="cuda")
    mask[3:5, 3:5, 6:9] = 1
    cells = np.array([[3, 2, 2], [15, 5, 7], [10, 3, 4], [20, 6, 8], [1, 1, 1]])
    uhat = torch.randn((len(cells), 3), device="cuda", generator=g)
    ref = ProbeProblem(p, cells, nsteps, blanking=mask, checkpoint=3)
    ru = ref.forward(f1, f2, uvel)
    rg, rv = ref.backward(uhat)
    a = FusedProbeProblem(p, cells, nsteps, blanking=mask, checkpoint=K)
    a.forward(f1 * 1.001, f2, uvel)              # another run's arrays are dropped
    for _ in range(2):
        u = a.forward(f1, f2, uvel)
        assert float((u - ru).abs().max()) < 1e-6
        end = [a.lbm.empty_s() for _ in range(4)]
        a.lbm.get_macro(*end)
        for overlap in (True, True, False, False):
            # the same sums in another order, some by atomics: within the two sweeps' distance (3e-5 of
            # the largest entry, test_gpu_adjoint.py)
            fg, fv = a.backward(uhat, overlap=overlap)
            assert float((fg - rg).abs().max()) < 1e-4 * float(rg.abs().max())
            assert float((fv - rv).abs().max()) < 1e-4 * float(rv.abs().max())
            if overlap:      # the forward's context still holds the state after the last step
                now = [a.lbm.empty_s() for _ in range(4)]
                a.lbm.get_macro(*now)
                assert all(torch.equal(x, y) for x, y in zip(now, end))
    assert float((a.forward(f1, f2, uvel, keep=False) - ru).abs().max()) < 1e-6
    a.close()
    ref.close()


@pytest.mark.parametrize("nsteps,K,nx", [(9, 4, 21), (13, 3, 23)])
def test_segments_of_odd_rows(nsteps, K, nx):
    test_segments_give_the_percall_gradient(nsteps, K, nx)


def small_problem(nsteps, K, nx=20):
    from lbm_b200 import Lbm, Params
    from lbm_b200.adjoint import FusedProbeProblem, initial_state
    p = Params(nx=nx, ny=8, nz=8, nl=19, iturb_pos=2)
    m = [torch.zeros(p.sshape, device="cuda") for _ in range(4)]
    m[0][1:-1, 1:-1, 1:-1] = 1.0
    uvel = torch.full((p.nz,), 0.05, device="cuda")
    with Lbm(p) as L:
        f1, f2 = initial_state(L, *m, uvel)
        torch.cuda.synchronize()
    cells = np.array([[3, 2, 2], [15, 5, 7], [10, 3, 4]])
    return FusedProbeProblem(p, cells, nsteps, checkpoint=K), f1, f2, uvel


@pytest.mark.parametrize("nsteps,K", [(6, 6), (12, 6), (15, 6), (18, 6)])
@pytest.mark.parametrize("overlap", [True, False])
def test_backward_gives_the_kept_states_back(nsteps, K, overlap):
    """After a gradient a problem holds its checkpoints and two states, whatever the number of
    segments; the arrays of the last segment and of the replays are free again."""
    a, f1, f2, uvel = small_problem(nsteps, K)
    uhat = torch.ones((3, 3), device="cuda")
    base = torch.cuda.memory_allocated()
    state = a.lbm.state_bytes()
    for _ in range(2):
        a.forward(f1, f2, uvel)
        for _ in range(2):
            a.backward(uhat, overlap=overlap)
            bound = 2 * state + sum(t.numel() * 4 for c in a.ckpt.values() for t in (c if isinstance(c, tuple) else (c,)))
            assert torch.cuda.memory_allocated() - base < bound + state // 2      # less than a third state
    a.close()
    assert torch.cuda.memory_allocated() - base < state // 2


@pytest.mark.parametrize("nsteps,K", [(6, 6), (9, 3), (14, 3)])
@pytest.mark.parametrize("overlap", [True, False])
def test_replay_arrays_are_made_before_the_adjoint_steps(nsteps, K, overlap, monkeypatch):
    """The replay stream is ordered behind what was queued when the sweep began, so an array
    made for it later could be memory that the adjoint stream has still to read."""
    a, f1, f2, uvel = small_problem(nsteps, K)
    uhat = torch.ones((3, 3), device="cuda")
    calls = []
    scratch, step = a.lbm.state_scratch, a.lbm.state_adjoint_step
    monkeypatch.setattr(a.lbm, "state_scratch", lambda: (calls.append("array"), scratch())[1])
    monkeypatch.setattr(a.lbm, "state_adjoint_step", lambda *x: (calls.append("step"), step(*x))[1])
    for _ in range(2):
        a.forward(f1, f2, uvel)
        for _ in range(2):
            calls.clear()
            a.backward(uhat, overlap=overlap)
            assert calls.count("step") == nsteps
            assert "array" not in calls[calls.index("step"):]
    a.close()


def test_the_context_keeps_its_state_after_a_serial_backward():
    """Without overlap the forward's own context replays; the arrays it ends on stay with it."""
    a, f1, f2, uvel = small_problem(13, 4)
    a.forward(f1, f2, uvel)
    a.backward(torch.ones((3, 3), device="cuda"), overlap=False)
    M = [torch.empty(a.p.sshape, device="cuda") for _ in range(4)]
    a.lbm.get_macro(*M)
    fill = [a.lbm.state_scratch().fill_(float("nan")) for _ in range(12)]       # whatever was given back
    N = [torch.empty(a.p.sshape, device="cuda") for _ in range(4)]
    a.lbm.get_macro(*N)
    assert all(torch.equal(x, y) for x, y in zip(M, N))
    del fill
    a.close()
