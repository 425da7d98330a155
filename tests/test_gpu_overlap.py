"""Steps of several contexts in flight at once, each context on its own stream, give each context
the bits of its lone run: contexts share no memory, and every kernel orders its refills of shared
memory by bulk copies after the reads they follow, however long those queue behind the other
contexts' loads. An odd number of quadrature nodes takes the general kernels: with odd nz the
stencil that reads psi by global loads while projection fragments come by bulk copies, with even
nz the staged one; an even number takes the octant kernels."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


class _Problem:
    """A gaussian pulse over a floor, two time steps from its start."""

    def __init__(self, torch, N, Q, n, width):
        T = c3d.quadrature(N, Q, with_m2=True)
        nm, nq = T["nm"], T["nq"]
        _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
        self.x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=2 / n[0], dy=2 / n[1],
                             dz=2 / n[2], M=T["M"], w=T["w"], xi=T["xi"], eta=T["eta"],
                             mu=T["mu"], tol=1e-6, ladder=(0.0, 1e-8, 1e-6, 1e-4, 1e-2, 1e-1))
        self.x.set_gaunt(T["nm2"], T["M2"], row, col, val)
        X = np.meshgrid(*[-1 + (np.arange(-2, e + 2) + 0.5) * 2 / e for e in n], indexing="ij")
        G = np.exp(-sum(v * v for v in X) / (2 * width ** 2)) / (width * np.sqrt(2 * np.pi)) ** 3
        u = np.zeros((G.size, nm))
        u[:, 0] = 2 * np.sqrt(np.pi) * np.maximum(1e-8, G.ravel() / (4 * np.pi))
        a = np.zeros_like(u)
        a[:, 0] = np.sqrt(4 * np.pi) * np.log(u[:, 0] / np.sqrt(4 * np.pi))
        self.u, self.a = torch.tensor(u, device="cuda"), torch.tensor(a, device="cuda")
        self.sig = torch.ones(G.size, dtype=torch.float64, device="cuda")
        self.uo, self.ao = torch.empty_like(self.u), torch.empty_like(self.a)
        self.dt = 0.25 / sum(e / 2 for e in n)

    def run(self):
        L, h, s = c3d.lib(), self.x.h, self.sig.data_ptr()
        c3d.check(L.c3d_set_state(h, self.u.data_ptr(), self.a.data_ptr(), s, s, 1), "set_state")
        for _ in range(2):
            self.x.step(self.dt)
        c3d.check(L.c3d_get_state(h, self.uo.data_ptr(), self.ao.data_ptr(), 1), "get_state")


@pytest.mark.parametrize("N,Q,n", [(3, 15, (37, 45, 51)), (3, 15, (37, 45, 50)), (2, 11, (29, 31, 33)),
                                   (5, 17, (23, 21, 27)), (3, 14, (37, 45, 51))])
def test_overlapped_steps_are_the_lone_steps(N, Q, n):
    import torch
    P = [_Problem(torch, N, Q, n, w) for w in (0.15, 0.13, 0.17)]
    torch.cuda.synchronize()
    lone = []
    for p in P:
        p.run()
        torch.cuda.synchronize()
        lone.append((p.uo.clone(), p.ao.clone()))
    torch.cuda.synchronize()
    wrong = 0
    for _ in range(30):
        for p in P:
            p.run()
        torch.cuda.synchronize()
        wrong += sum(not (torch.equal(p.uo, u) and torch.equal(p.ao, a)) for p, (u, a) in zip(P, lone))
    for p in P:
        p.x.sync()
        p.x.close()
    assert wrong == 0
