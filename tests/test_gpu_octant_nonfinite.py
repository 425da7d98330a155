"""Infinities and NaNs in the octant kernels. A transform over the 8 reflections turns one infinite
direction into NaNs of all parity classes, where the general kernels have infinities in some sums.
The closure's decisions do not see the difference: the objective stays infinite and a factorisation
of either kind fails, so such a cell restarts from isotropy or backtracks in both. The flux of a cell
next to an overflowing one is not finite in both, and all other values agree.

Both contexts hold the same directions, in the tensor order (octant kernels) and rotated (general
ones). Tolerances as between the two on ordinary values: 1e-13 for a flux, 1e-12 and 1e-9 for closed
moments and multipliers, equal iterations at tolerance 1e-6."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


def _contexts(N, Q, n, **kw):
    T = c3d.quadrature(N, Q, with_m2=True)
    nm, nq = T["nm"], T["nq"]
    M = T["M"].reshape(nq, nm)
    _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
    out = []
    for shift in (0, 1):
        t = {k: np.roll(T[k], shift) for k in ("w", "xi", "eta", "mu")}
        x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=nq, dx=2 / n[0], dy=2 / n[1],
                        dz=2 / n[2], M=np.roll(M, shift, axis=0).ravel(), tol=1e-6,
                        ladder=(0.0, 1e-8, 1e-6, 1e-4, 1e-2, 1e-1), **t, **kw)
        M2 = np.roll(T["M2"].reshape(nq, -1), shift, axis=0)
        x.set_gaunt(T["nm2"], M2.ravel(), row, col, val)
        assert x.octant_info()[:2] == (shift == 0, shift == 0)
        out.append(x)
    return T, out


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("N,Q,n", [(1, 8, (9, 8, 10)), (3, 12, (10, 9, 11)), (6, 18, (8, 8, 8))])
def test_flux_next_to_an_overflow(N, Q, n):
    T, ctxs = _contexts(N, Q, n)
    nm = T["nm"]
    full = tuple(e + 4 for e in n)
    nall = full[0] * full[1] * full[2]
    rng = np.random.default_rng([3, N])
    a = rng.standard_normal((nall, nm)) * 0.2
    cell = np.ravel_multi_index((5, 6, 5), full)
    # exponents 705 +- 20 or more: some directions overflow, others do not
    a[cell, 0] = 705 * 2 * np.sqrt(np.pi)
    a[cell, 1:] = rng.choice([-1.0, 1.0], nm - 1) * 60.0 / np.sqrt(nm)
    z = T["M"].reshape(T["nq"], nm) @ a[cell]
    assert (z > 710).any() and (z < 705).any()
    f = []
    for x in ctxs:
        x.set_state(u=a.ravel(), alpha=a.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        x.flux_kinetic(0)
        x.sync()
        f.append(x.get_flux().reshape(nall, nm))
        x.close()
    bad = [~np.isfinite(v).all(axis=1) for v in f]
    assert bad[0][cell] and np.array_equal(bad[0], bad[1])
    # values up to 1e308 beside the overflow would drown the rest: compare per cell
    ok = ~bad[0] & (np.abs(f[1]).max(axis=1) > 0)
    scale = np.abs(f[1][ok]).max(axis=1, keepdims=True)
    assert (np.abs(f[0][ok] - f[1][ok]) / scale).max() < 1e-12


@pytest.mark.parametrize("N,Q", [(1, 8), (3, 12), (5, 16), (6, 18)])
@pytest.mark.parametrize("mode", [0, 1])
def test_cells_that_overflow_restart(N, Q, mode):
    n = (6, 5, 4)
    T, ctxs = _contexts(N, Q, n)
    nm, nq = T["nm"], T["nq"]
    nall = 10 * 9 * 8
    M = T["M"].reshape(nq, nm)
    rng = np.random.default_rng([4, N])
    a = rng.standard_normal((nall, nm)) * 0.3
    a[:, 0] = 0.0
    u = (np.exp(a @ M.T) * T["w"]) @ M
    start = a + 0.1 * rng.standard_normal((nall, nm))
    # scaled exponents beyond 710 in some directions (multipliers of norm below 32, so the symmetric
    # passes form them), in all of them, and a NaN
    c = rng.choice(nall, 30, replace=False)
    u[c] *= 1e-300 / u[c, :1]
    start[c[:15], 0] = (709.5 + np.log(1e-300) + np.log(2 * np.sqrt(np.pi))) * 2 * np.sqrt(np.pi)
    start[c[:15], 1:] = rng.standard_normal((15, nm - 1)) * 0.5
    start[c[15:25], 0] = 300.0
    start[c[25:], nm - 1] = np.nan
    res = []
    for x in ctxs:
        x.set_precision(mode)
        x.set_state(u=u.ravel(), alpha=start.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        x.closure()
        x.sync()
        res.append(x.get_state() + (x.records(),))
        x.close()
    (u0, a0, r0), (u1, a1, r1) = res
    for k in ("iters", "regIndex", "status"):
        assert np.array_equal(r0[k], r1[k]), k
    assert not r0["status"].any() and (r0["iters"][c] > 1).all()
    assert np.isfinite(a0).all() and np.isfinite(u0).all()
    s0, s1 = (v.reshape(nall, nm) / v.reshape(nall, nm)[:, :1] for v in (u0, u1))
    assert _rel(s0, s1) < (1e-12 if mode == 0 else 1e-10)
    assert _rel(a0, a1) < (1e-9 if mode == 0 else 1e-8)
