"""The octant-symmetric kernels against the general ones. The tensor quadrature in its own
order takes the symmetric kernels; the same directions in a rotated order are not recognised as
symmetric and take the general ones, which the other tests check against the oracle. Both
compute the same sums in another order.

Tolerances: a flux value is a sum of nq terms whose rounding errors are a few ulps of psi, so
1e-13 relative L2 as for the flux everywhere in these tests; a closed cell's moments are those of
the stopping test, so the moments of a step agree to 1e-12 and its multipliers to 1e-9 (condition
numbers up to 1e6 here); iteration counts are equal (no rounding ties at tolerance 1e-6).

Sizes: octant directions that fill no block of 8 or group of 4 (Q = 10: 25, Q = 14: 49), one
block exactly (Q = 8: 16 = 2 blocks), tiles of the stencil (4 x 4 x 8) exact, ragged and larger
than the grid, odd z edges (8-byte copies), and a psi budget that splits the directions."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


def _contexts(N, Q, n, gaunt=False, **kw):
    T = c3d.quadrature(N, Q, with_m2=gaunt)
    nm, nq = T["nm"], T["nq"]
    M = T["M"].reshape(nq, nm)
    if gaunt:
        _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
    out = []
    for shift in (0, 1):
        t = {k: np.roll(T[k], shift) for k in ("w", "xi", "eta", "mu")}
        x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=2 / n[0], dy=2 / n[1],
                        dz=2 / n[2], M=np.roll(M, shift, axis=0).ravel(), tol=1e-6, **t, **kw)
        if gaunt:
            M2 = np.roll(T["M2"].reshape(nq, -1), shift, axis=0)
            x.set_gaunt(T["nm2"], M2.ravel(), row, col, val)
        out.append(x)
    return T, out


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("N,Q,n,chunk", [
    (0, 2, (3, 2, 1), 0), (1, 8, (8, 8, 8), 0), (2, 10, (9, 5, 7), 0), (3, 14, (4, 12, 33), 0),
    (4, 12, (13, 17, 24), 96), (5, 16, (16, 16, 16), 0), (6, 18, (11, 4, 10), 160),
    (7, 20, (5, 9, 9), 0)])
@pytest.mark.parametrize("theta,pn", [(2.0, 0), (1.0, 0), (2.0, 1)])
def test_flux_matches_general_kernels(N, Q, n, chunk, theta, pn):
    nall = (n[0] + 4) * (n[1] + 4) * (n[2] + 4)
    kw = dict(theta=theta, psi_bytes=chunk * nall * 8)
    if pn:
        kw.update(solver=0, pn_kinetic=1)
    T, ctxs = _contexts(N, Q, n, **kw)
    rng = np.random.default_rng([N, Q, pn])
    a = rng.standard_normal((nall, T["nm"])) * 0.3
    f = []
    for x in ctxs:
        x.set_state(u=a.ravel(), alpha=a.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        x.flux_kinetic(pn)
        x.sync()
        f.append(x.get_flux())
        x.close()
    assert np.isfinite(f[0]).all()
    assert _rel(f[0], f[1]) < 1e-13


@pytest.mark.parametrize("N,Q,n", [(0, 4, (20, 20, 24)), (2, 10, (18, 22, 26)), (4, 12, (35, 34, 36)),
                                   (6, 14, (21, 24, 17)), (7, 16, (17, 19, 25))])
def test_flux_on_wider_tiles(N, Q, n):
    """Grids whose stencil takes tiles of 4 x planes (a wave of them or more on 148 SMs), their last
    tiles ragged along x, y and z."""
    test_flux_matches_general_kernels(N, Q, n, 0, 2.0, 0)


@pytest.mark.parametrize("N,Q,n", [(1, 8, (8, 6, 5)), (2, 10, (12, 9, 8)), (3, 14, (10, 12, 11)),
                                   (4, 14, (8, 8, 16)), (5, 16, (9, 8, 10)), (6, 18, (8, 8, 8)),
                                   (7, 20, (6, 6, 6))])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("graphs", [True, False])
def test_steps_match_general_kernels(N, Q, n, mode, graphs):
    T, ctxs = _contexts(N, Q, n, gaunt=True, ladder=(0.0, 1e-8, 1e-6, 1e-4, 1e-2, 1e-1))
    nm = T["nm"]
    full = tuple(e + 4 for e in n)
    nall = full[0] * full[1] * full[2]
    # a smooth periodic field with warm starts a few per cent off: every cell iterates
    g = [(np.arange(-2, e + 2) + 0.5) * 2 * np.pi / e for e in n]
    X = np.meshgrid(*g, indexing="ij")
    rng = np.random.default_rng([7, N])
    a = np.zeros((nall, nm))
    for m in range(nm):
        ph = rng.uniform(0, 6, 3)
        amp = 1.5 if m == 0 else 0.4 * 0.7 ** np.sqrt(m)
        a[:, m] = amp * (np.cos(X[0] + ph[0]) * np.cos(X[1] + ph[1]) * np.cos(X[2] + ph[2])).ravel()
    M = T["M"].reshape(T["nq"], nm)
    u = (np.exp(a @ M.T) * T["w"]) @ M
    start = a * (1 + 0.03 * np.sin(X[0]).reshape(-1, 1))
    dt = 0.25 / sum(e / 2 for e in n)
    res = []
    for x in ctxs:
        x.set_precision(mode)
        x.set_graphs(graphs)
        x.set_state(u=u.ravel(), alpha=start.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        x.step(dt)
        x.sync()
        res.append(x.get_state() + (x.records(), x.stats().totalIters))
        x.close()
    (u0, a0, r0, t0), (u1, a1, r1, t1) = res
    assert t0 > 2 * nall  # Newton steps, not only certified first visits
    # mixed: reduced-precision Hessians amplify a last-bit difference to the stopping tolerance
    # times the Newton contraction, far below the mixed closure's own 1e-8
    assert _rel(u0, u1) < (1e-12 if mode == 0 else 1e-10)
    assert _rel(a0, a1) < (1e-9 if mode == 0 else 1e-8)
    for k in ("iters", "regIndex", "status"):
        assert np.array_equal(r0[k], r1[k]), k
    assert t0 == t1


@pytest.mark.parametrize("N,Q,n", [(6, 28, (20, 20, 20)), (6, 28, (22, 20, 22))])
def test_cells_at_the_realizability_boundary(N, Q, n):
    """Two steps of a narrow pulse over a low floor: its edge cells reach multipliers in the
    hundreds and take their passes in the reference's order (over all directions, so rotating
    them changes the sums' rounding only). Amplified by condition numbers to 1e9 that moves a
    cell's multipliers by up to 1e-7 inside the stopping tolerance (1e-6 on the scaled gradient)
    and its moments' update by the same order; 1e-6 relative L2 on the grid bounds both, and no
    cell fails."""
    T, ctxs = _contexts(N, Q, n, gaunt=True, ladder=(0.0, 1e-8, 1e-6, 1e-4, 1e-2, 1e-1))
    nm = T["nm"]
    x = [-1 + (np.arange(-2, e + 2) + 0.5) * 2 / e for e in n]
    X = np.meshgrid(*x, indexing="ij")
    s = 0.02
    G = np.exp(-sum(v * v for v in X) / (2 * s * s)) / (s * np.sqrt(2 * np.pi)) ** 3
    u = np.zeros((G.size, nm))
    u[:, 0] = 2 * np.sqrt(np.pi) * np.maximum(1e-10, G.ravel() / (4 * np.pi))
    a = np.zeros_like(u)
    a[:, 0] = np.sqrt(4 * np.pi) * np.log(u[:, 0] / np.sqrt(4 * np.pi))
    dt = 0.25 / sum(e / 2 for e in n)
    res, far = [], 0
    for c in ctxs:
        c.set_state(u=u.ravel(), alpha=a.ravel(), sig_t=np.ones(G.size), sig_s=np.ones(G.size))
        for _ in range(2):
            c.step(dt)
        c.sync()
        uu, aa = c.get_state()
        far = max(far, np.linalg.norm(aa.reshape(-1, nm)[:, 1:], axis=1).max())
        res.append((uu, aa, c.records()["status"]))
        c.close()
    assert far > 32.0  # cells on the reference-order list
    assert not res[0][2].any() and not res[1][2].any()
    assert _rel(res[0][0], res[1][0]) < 1e-6
    assert _rel(res[0][1], res[1][1]) < 1e-6


@pytest.mark.parametrize("N", [3, 4, 5])
def test_regularised_cells_match_persistent_engine(N):
    """Cells far from isotropy under a condition limit of 200: isotropic restarts and several
    ladder levels, which read a cell's start and original vectors again -- orders up to 4 from its
    global state, N = 5 and the persistent engine from the slot. Both engines take the same
    decisions (no ties at tolerance 1e-6: the condition estimates agree to 1e-12); rounding
    amplified by condition numbers up to 200 over some ten iterations stays below 1e-9."""
    n, Q = (9, 8, 7), 2 * (N + 3)
    T = c3d.quadrature(N, Q, with_m2=True)
    nm, nq = T["nm"], T["nq"]
    _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
    nall = (n[0] + 4) * (n[1] + 4) * (n[2] + 4)
    M = T["M"].reshape(nq, nm)
    rng = np.random.default_rng([11, N])
    a = rng.standard_normal((nall, nm)) * rng.uniform(0.2, 1.5, (nall, 1))
    a[:, 0] = 0.0
    u = (np.exp(a @ M.T) * T["w"]) @ M
    start = np.zeros_like(a)
    start[:, 0] = 2 * np.sqrt(np.pi) * np.log(u[:, 0] / (2 * np.sqrt(np.pi)))
    res = []
    for engine in (0, 1):
        x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=1.0, dy=1.0, dz=1.0, M=T["M"],
                        w=T["w"], xi=T["xi"], eta=T["eta"], mu=T["mu"], tol=1e-6, cond_h_max=200.0,
                        ladder=(0.0, 1e-2, 1e-1, 0.5, 0.9, 0.99))
        x.set_gaunt(T["nm2"], T["M2"], row, col, val)
        x.set_engine(engine)
        x.set_state(u=u.ravel(), alpha=start.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        x.closure()
        x.sync()
        res.append(x.get_state() + (x.records(),))
        x.close()
    (u0, a0, r0), (u1, a1, r1) = res
    assert len(set(r0["regIndex"])) >= 3 and (r0["regIndex"] > 0).sum() > 20
    for k in ("iters", "regIndex", "status"):
        assert np.array_equal(r0[k], r1[k]), k
    assert _rel(u0, u1) < 1e-9 and _rel(a0, a1) < 1e-9
