"""Grids with an axis of one cell. The image of a ghost layer is then a ghost layer itself: the
reference's exchange copies layer by layer, so the outer low layer takes what the inner one held
before (src/comm.cpp:281-323). Steps agree with the oracle: no ghost copy races with another, and
the flux reads no face ghost's ansatz that the closure left out.

Tolerances: P_N steps are sums of the oracle's terms in another order (1e-13 relative L2), M_N
steps too where every cell takes the oracle's decisions (no ties at tolerance 1e-6; at 1e-8 single
rounding errors decide): moments within 1e-12 a step, multipliers within 1e-9 (condition numbers up
to 1e6)."""
import numpy as np
import pytest

import c3d
from oracle_lib import make_opts

from test_gpu_kernels import _gaunt_csr

pytestmark = pytest.mark.gpu

GRIDS = [(6, 5, 1), (1, 6, 5), (5, 1, 6), (1, 1, 4), (1, 1, 1)]


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _start(n, nm):
    X = np.meshgrid(*[-1 + (np.arange(-2, e + 2) + 0.5) * 2 / e for e in n], indexing="ij")
    G = 0.1 + np.exp(-sum(v * v for v in X) / 0.5)
    u = np.zeros((G.size, nm))
    u[:, 0] = 2 * np.sqrt(np.pi) * G.ravel()
    a = np.zeros_like(u)
    a[:, 0] = 2 * np.sqrt(np.pi) * np.log(u[:, 0] / (2 * np.sqrt(np.pi)))
    return u.ravel(), a.ravel()


@pytest.mark.parametrize("n", GRIDS)
def test_ghost_fill_is_the_reference_exchange(oracle, n):
    T = oracle.tables(1, 6)
    nm, nq = T["nm"], T["nq"]
    g = oracle.grid(*n, nm, nq, 1.0, 1.0, 1.0, 2.0)
    x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=1.0, dy=1.0, dz=1.0, M=T["M"],
                    w=T["w"], xi=T["xi"], eta=T["eta"], mu=T["mu"])
    u = np.random.default_rng(1).standard_normal((n[0] + 4) * (n[1] + 4) * (n[2] + 4) * nm)
    x.set_state(u=u)
    for _ in range(2):
        x.ghost_fill()
        oracle.ghost_fill(g, u)
        assert np.array_equal(x.get_state()[0], u)
    x.close()


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("Q", [10, 11])
@pytest.mark.parametrize("graphs", [True, False])
def test_mn_steps_match_oracle(oracle, n, Q, graphs):
    T = oracle.tables(2, Q, gaunt=True)
    nm, nq = T["nm"], T["nq"]
    d = [2 / e for e in n]
    row, col, val = _gaunt_csr(T, 1e-13)
    x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=d[0], dy=d[1], dz=d[2], M=T["M"],
                    w=T["w"], xi=T["xi"], eta=T["eta"], mu=T["mu"], tol=1e-6)
    x.set_gaunt(T["nm2"], T["M2"], row, col, val)
    x.set_graphs(graphs)
    u, a = _start(n, nm)
    sig = np.ones(len(u) // nm)
    x.set_state(u=u, alpha=a, sig_t=sig, sig_s=sig)
    g = oracle.grid(*n, nm, nq, *d, 2.0)
    opts = make_opts(nm, nq, nm2=T["nm2"], hess_mode=2, tol=1e-6)
    dt = 0.2 / sum(1 / e for e in d)
    for _ in range(3):
        x.step(dt)
        oracle.step(g, opts, T, u, a, sig, sig, dt, records=False)
    x.sync()
    ug, ag = x.get_state()
    x.close()
    assert _rel(ug, u) < 3e-12 and _rel(ag, a) < 1e-9


@pytest.mark.parametrize("n", GRIDS)
def test_pn_steps_match_oracle(oracle, n):
    T = oracle.tables(3, 8, pn=True)
    nm, nq = T["nm"], T["nq"]
    d = [2 / e for e in n]
    x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=d[0], dy=d[1], dz=d[2], M=T["M"],
                    w=T["w"], xi=T["xi"], eta=T["eta"], mu=T["mu"], solver=0, pn_ops=T["pnops"])
    u, _ = _start(n, nm)
    sig = np.ones(len(u) // nm)
    x.set_state(u=u, sig_t=sig, sig_s=sig)
    g = oracle.grid(*n, nm, nq, *d, 2.0)
    dt = 0.1 / sum(1 / e for e in d)
    for _ in range(4):
        x.step(dt)
        oracle.step(g, make_opts(nm, nq), T, u, np.zeros_like(u), sig, sig, dt, solver=0, records=False)
    x.sync()
    ug, _ = x.get_state()
    x.close()
    assert _rel(ug, u) < 1e-13
