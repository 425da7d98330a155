"""Fused trials (closure_rounds.cu): the pass of a line-search trial also forms the moments at the
trial point, and the next Hessian visit takes them when -- and only when -- the trial is accepted.

A mixed-precision cell whose line search backtracks to the end after a reduced-precision Hessian
goes back to the multipliers before the trial and redoes the iteration with FP64 moments, which
belong to those multipliers: it needs a pass of its own. Vectors that start converged, under a
tolerance no gradient meets, end their first line search that way or accept a rounding-level step.
Each is solved alone with host-driven rounds, one pass per round, so the rounds count the passes:
one per reduced-precision Hessian visit, one per trial and one per redone iteration; a Hessian
visit after an accepted trial has none."""
import numpy as np
import pytest

import c3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [3, 4, 5])
def test_redone_iteration_takes_its_own_moments(N):
    import torch
    Q, n = 2 * (N + 3), 48
    T = c3d.quadrature(N, Q, with_m2=True)
    nm, nq = T["nm"], T["nq"]
    _, row, col, val = c3d.gaunt_build(nm, T["nm2"], nq, T["M2"])
    M = T["M"].reshape(nq, nm)
    rng = np.random.default_rng([5, N])
    a = rng.standard_normal((n, nm)) * 0.3
    u = (np.exp(a @ M.T) * T["w"]) @ M
    x = c3d.Context(nx=2, ny=2, nz=2, nm=nm, nq=nq, dx=1.0, dy=1.0, dz=1.0, M=T["M"], w=T["w"],
                    xi=T["xi"], eta=T["eta"], mu=T["mu"], tol=1e-18, ladder=(0.0,),
                    max_iter=4)
    x.set_gaunt(T["nm2"], T["M2"], row, col, val)
    # every Hessian after a cell's first (3xTF32) one is FP64, and so are its trials' moments
    x.set_precision(1, cond_bf16=1e-6, cond_mixed_max=1e-6, polish=1.0)
    x.set_graphs(False)
    redone = 0
    for i in range(n):
        ud = torch.tensor(u[i], device="cuda")
        ad = torch.tensor(a[i], device="cuda")
        torch.cuda.synchronize()
        x.reset_stats()
        before = x.stats().hostSyncs
        x.closure_vectors_device(1, ud.data_ptr(), ad.data_ptr())
        try:
            x.sync()
        except c3d.C3DError:
            pass  # the line search of the last iteration fails: the one-level ladder is exhausted
        s = x.stats()
        rounds = s.hostSyncs - before - 1  # the last wait finds the lists empty
        assert s.hessTf32x3 == 1 and s.escalated <= 1
        assert rounds == s.hessTf32x3 + s.trials + s.escalated, (i, rounds, s.trials, s.escalated)
        redone += s.escalated
    x.close()
    assert redone > 0
