"""c3d_launch_count counts the hand-off's kernels: with it a closure issues the marks' groups, the
refresh of the marked cells and, mirrored, the face ghosts' copy on top of a closure without."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q", [8, 9])
@pytest.mark.parametrize("mirror", [True, False])
@pytest.mark.parametrize("graphs", [True, False])
def test_handoff_launches_are_counted(Q, mirror, graphs):
    T = c3d.quadrature(2, Q, with_m2=True)
    nm, nq, n = T["nm"], T["nq"], 6
    _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
    nall = (n + 4) ** 3
    u = np.zeros((nall, nm))
    u[:, 0] = 1.0
    a = np.zeros_like(u)
    a[:, 0] = 2 * np.sqrt(np.pi) * np.log(1.0 / (2 * np.sqrt(np.pi)))
    count = {}
    for handoff in (True, False):
        x = c3d.Context(nx=n, ny=n, nz=n, nm=nm, nq=nq, dx=1.0, dy=1.0, dz=1.0, M=T["M"], w=T["w"],
                        xi=T["xi"], eta=T["eta"], mu=T["mu"], tol=1e-6)
        x.set_gaunt(T["nm2"], T["M2"], row, col, val)
        x.set_graphs(graphs)
        x.set_ghost_mirroring(mirror)
        x.set_ansatz_handoff(handoff)
        x.set_state(u=u.ravel(), alpha=a.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        before = x.launch_count()
        x.closure()
        x.sync()
        count[handoff] = x.launch_count() - before
        x.close()
    assert count[True] - count[False] == (3 if mirror else 2)
