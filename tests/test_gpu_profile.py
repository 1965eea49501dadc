"""Step timing over more steps than the context keeps events for: the recorded triples are
drained and used again."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [681, 682, 683, 1500])
def test_profile_of_many_steps(steps):
    from lbm_b200 import Params, Solver
    p = Params(nx=8, ny=4, nz=4, nl=19, iturb_pos=2)
    m = [torch.zeros(p.sshape, device="cuda") for _ in range(4)]
    m[0][1:-1, 1:-1, 1:-1] = 1.0
    s = Solver(p, *m, torch.full((p.nz,), 0.05, device="cuda"))
    s.step(1)                    # the first step collides in place and is not timed
    s.lbm.profile(True)
    s.step(steps)
    ms, n = s.lbm.profile_read()
    bc, nb = s.lbm.profile_read_boundary()
    s.lbm.profile(False)
    assert n == steps and nb == steps and ms > 0.0 and bc > 0.0
    assert s.lbm.status() == 0
