"""The P_N moment flux against the formula in numpy (src/flux_moment.cpp:57-101), for every
moment order (1 to 8 tiles of 8 moments, with and without padding), grids of one cell, of one
partial tile of cells, of both cell widths of the kernel's dispatch, and unequal spacings.

Tolerance: a value is 6 sums of nm products of O(1) factors, each product and sum rounded once;
random rounding gives about sqrt(6 nm) eps relative, 1e-14 at nm = 64; 1e-13 relative L2 as for
the flux everywhere in these tests."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [(0, (1, 1, 1)), (1, (3, 2, 4)), (2, (9, 7, 5)), (3, (8, 8, 8)),
                                 (4, (5, 6, 11)), (5, (37, 33, 35)), (6, (4, 9, 3)),
                                 (7, (34, 35, 36))])
def test_moment_flux_matches_numpy(N, n):
    nm = (N + 1) ** 2
    T = c3d.quadrature(N, 2 * (N + 1))
    rng = np.random.default_rng([3, N])
    ops = rng.standard_normal((6, nm, nm)) / nm
    h = (0.1, 0.25, 0.4)
    x = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=nm, nq=T["nq"], dx=h[0], dy=h[1], dz=h[2],
                    M=T["M"], w=T["w"], xi=T["xi"], eta=T["eta"], mu=T["mu"], solver=0,
                    pn_ops=ops.ravel())
    full = tuple(e + 4 for e in n)
    u = rng.standard_normal(full + (nm,))
    sig = np.ones(full).ravel()
    x.set_state(u=u.ravel(), sig_t=sig, sig_s=sig)
    x.flux_moment()
    x.sync()
    f = x.get_flux().reshape(full + (nm,))
    x.close()
    want = 0.0
    for ax in range(3):
        v = u
        for other in range(3):
            if other != ax:
                v = np.take(v, range(2, 2 + n[other]), axis=other)
        m2, m1, v0, p1, p2 = (np.take(v, range(k, k + n[ax]), axis=ax) for k in range(5))
        tp = 0.25 * p1 + 0.75 * v0 - 1.25 * m1 + 0.25 * m2
        tm = -0.25 * p2 + 1.25 * p1 - 0.75 * v0 - 0.25 * m1
        want = want + (tp @ ops[2 * ax].T + tm @ ops[2 * ax + 1].T) / h[ax]
    got = f[2:-2, 2:-2, 2:-2]
    assert np.linalg.norm(got - want) < 1e-13 * np.linalg.norm(want)
    f[2:-2, 2:-2, 2:-2] = 0.0
    assert not f.any()  # ghosts untouched
