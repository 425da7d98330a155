"""Which kernels run (c3d_octant_info): every even tensor quadrature in its own order takes the
octant-symmetric kernels in the flux and, in the Gaunt form, in the closure; odd numbers of nodes,
another order of the directions and a beta table whose column 0 is not m_0 mom_i take the general
ones. And the list of cells far out, whose passes keep the reference's order, holds the cells near
the realizability boundary: their multipliers agree with the oracle's per cell."""
import ctypes
import os

import numpy as np
import pytest

import c3d
from oracle_lib import deck_text, make_opts, tie_cells

pytestmark = pytest.mark.gpu


def _context(N, Q, shift=0, gaunt=True, spoil=False):
    T = c3d.quadrature(N, Q, with_m2=True)
    nm, nq = T["nm"], T["nq"]
    t = {k: np.roll(T[k], shift) for k in ("w", "xi", "eta", "mu")}
    x = c3d.Context(nx=2, ny=2, nz=2, nm=nm, nq=nq, dx=1.0, dy=1.0, dz=1.0,
                    M=np.roll(T["M"].reshape(nq, nm), shift, axis=0).ravel(), **t)
    if gaunt:
        _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
        if spoil:
            val = val.copy()
            val[row[1]] *= 1.0 + 1e-9  # beta of element (0, 1): column 0 is no longer m_0 mom_i
            val[row[nm]] *= 1.0 + 1e-9  # and of (1, 0)
        x.set_gaunt(T["nm2"], np.roll(T["M2"].reshape(nq, -1), shift, axis=0).ravel(), row, col, val)
    return x


@pytest.mark.parametrize("N", range(8))
def test_even_quadratures_take_the_octant_kernels(N):
    for Q in sorted({2, 4, 8, 2 * (N + 1), 2 * (N + 3), 4 * N + 4, 28}):
        if Q < 2 * N + 1:
            continue  # too few nodes to tell the products' harmonics apart: beta is not Gaunt's
        x = _context(N, Q)
        assert x.octant_info() == (True, True, 0), Q
        x.set_engine(1)
        assert x.octant_info()[:2] == (True, False)
        x.close()


def test_other_directions_take_the_general_kernels():
    for args, info in (((2, 11), (False, False)), ((2, 10, 1), (False, False)),
                       ((2, 10, 0, False), (True, False)), ((2, 10, 0, True, True), (True, False))):
        x = _context(*args)
        assert x.octant_info()[:2] == info, args
        x.close()


def test_far_cells_match_the_oracle(oracle, tmp_path):
    """Three steps of the 20^3 M_6 pulse, whose edge cells pass through multipliers of norm above 32: the
    cells of every closure that iterate agree with the oracle to 1e-8 per cell (2e-9 at most in the
    reference's order; where the symmetric passes form those cells' sums, 9e-8), and their visits
    were on the list of that order."""
    n, tol, ladder = 20, 1e-6, [0.0, 1e-8, 1e-6, 1e-4, 1e-2, 1e-1]
    deck = tmp_path / "input.deck"
    deck.write_text(deck_text(NX=n, NY=n, NZ=n, MOMENT_ORDER=6, QUAD_ORDER=28, CFL_FACTOR=0.5,
                              CROSS_SECTION=1.0, INIT_FLOOR=1e-10, GAUSS_SIGMA=0.02,
                              INIT_COND="gaussian_psi", THETA=2.0, MN_TOL=tol,
                              MN_BATCHED="true", MN_USE_GAUNT_COEF="true",
                              MN_USE_GAUNT_SPARSE="true", REG_LADDER=",".join(map(str, ladder)),
                              OMP_THREADS=os.cpu_count() or 1))
    s = c3d.Solver(str(deck))
    L, ctx, nm = c3d.lib(), s.ctx_handle, s.nm
    T = oracle.tables(6, 28, gaunt=True)
    g = oracle.grid(n, n, n, nm, s.nq, s.dx, s.dy, s.dz, s.theta)
    opts = make_opts(nm, s.nq, nm2=T["nm2"], hess_mode=2, tol=tol, ladder=ladder)
    u, a = np.empty(s.nall * nm), np.empty(s.nall * nm)
    ptr = [v.ctypes.data_as(ctypes.c_void_p) for v in (u, a)]
    visits, far, checked = 0, 0, 0
    for step in range(3):
        for stage in range(2):
            c3d.check(L.c3d_get_state(ctx, *ptr, 0), "get_state")
            oracle.ghost_fill(g, u)
            u0, a0 = u.reshape(-1, nm).copy(), a.reshape(-1, nm).copy()
            c3d.check(L.c3d_closure_stats_reset(ctx), "reset")
            c3d.check(L.c3d_stage(ctx, stage, s.max_dt), "c3d_stage")
            s.sync()
            v = ctypes.c_longlong()
            c3d.check(L.c3d_octant_info(ctx, None, None, ctypes.byref(v)), "octant_info")
            visits += v.value
            c3d.check(L.c3d_get_state(ctx, *ptr, 0), "get_state")
            ag, rec = a.reshape(-1, nm), s.records()
            far += int((np.linalg.norm(ag[:, 1:], axis=1) > 32.0).sum())
            pick = np.nonzero(rec["iters"] > 1)[0]
            if len(pick) == 0:
                continue
            uo, ao = u0[pick], a0[pick]
            out = oracle.closure(opts, T, uo, ao)
            ok = ~tie_cells(out)
            assert np.array_equal(rec["iters"][pick][ok], out["totalIter"][ok])
            rel = np.linalg.norm(ag[pick][ok] - ao[ok], axis=1) / np.linalg.norm(ao[ok], axis=1)
            assert rel.max() < 1e-8, (step, stage, rel.max())
            checked += int(ok.sum())
    s.close()
    assert checked > 500 and far > 20 and visits >= far
