"""The certificate of the octant probe ends a cell only where the full visit would: its |g| is a sum
in another order than the full visit's, so a cell whose |g| lies at the tolerance up to rounding is
left to the full visit. Isotropic cells of M_1 have |g| of 0 to 4 ulps of 1; a tolerance of that
size puts them on either side of the stopping test by rounding alone, and runs with and without the
certificate still take the same iterations."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tol", [1.5e-16, 4e-16, 8e-16, 1e-6])
def test_cells_at_the_tolerance_take_the_full_visit(tol):
    T = c3d.quadrature(1, 8, with_m2=True)
    nm, nq, n = T["nm"], T["nq"], 6
    _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
    nall = (n + 4) ** 3
    rng = np.random.default_rng(3)
    u = np.zeros((nall, nm))
    u[:, 0] = np.exp(rng.uniform(-12, 3, nall))
    a = np.zeros_like(u)
    a[:, 0] = 2 * np.sqrt(np.pi) * np.log(u[:, 0] / (2 * np.sqrt(np.pi)))
    out = {}
    for on in (True, False):
        x = c3d.Context(nx=n, ny=n, nz=n, nm=nm, nq=nq, dx=1.0, dy=1.0, dz=1.0, M=T["M"], w=T["w"],
                        xi=T["xi"], eta=T["eta"], mu=T["mu"], tol=tol, max_iter=5)
        x.set_gaunt(T["nm2"], T["M2"], row, col, val)
        x.set_certificate(on)
        x.set_state(u=u.ravel(), alpha=a.ravel(), sig_t=np.ones(nall), sig_s=np.ones(nall))
        x.closure()
        try:
            x.sync()
        except c3d.C3DError:
            pass  # cells that no tolerance of this size lets converge exhaust the ladder
        out[on] = x.get_state() + (x.records(), x.stats().certified)
        x.close()
    for k in ("iters", "regIndex", "status"):
        assert np.array_equal(out[True][2][k], out[False][2][k]), k
    assert (out[True][3] > 0) == (tol > 1e-10)
    assert np.array_equal(out[True][0], out[False][0]) and np.array_equal(out[True][1], out[False][1])
