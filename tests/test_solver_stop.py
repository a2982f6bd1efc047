"""Where a saddle solve stops: at the first iterate whose residual is within the caller's tolerance."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsd_b200.configs import suspension
from fsd_b200.core import FSD

N = 200


@pytest.mark.gpu
@pytest.mark.parametrize("form", [dict(precond="ichol"), dict(precond="learned", learned_inner=4)],
                         ids=["ichol", "learned"])
@pytest.mark.parametrize("j", [6, 13, 20])
def test_solve_stops_at_the_first_iterate_within_tolerance(cuda, form, j):
    """Cycles of j - 1 and j iterations give the residuals r' > r of those iterates; a solve to a tolerance between
    them, at most 15 % above r, takes j iterations.  (Residuals of 1e-1 to 1e-5 here: the FP64 estimate that decides
    follows the true one to well within the 2 % that the two sides are kept apart.)"""
    pos, Lc = suspension(N, 0.3, 4)
    p = torch.as_tensor(pos).cuda().view(-1).contiguous()
    rhs = torch.as_tensor(np.random.default_rng(j).standard_normal(17 * N).astype(np.float32)).cuda()

    def solve(**kw):
        s = FSD(N, (Lc, Lc, Lc, 0.0), lanczos_max=4, **form, **kw)
        s.build_neighbor_list(p)
        s.precond_build(p)
        x, it, res, _ = s.saddle_solve(p, rhs, raise_on_error=False)
        s.close()
        return it, res

    # a tolerance below what FP32 reaches: the cycle is full, and max_iter ends the solve
    (it0, r0), (it1, r1) = (solve(solver_tol=1e-12, gmres_restart=k, gmres_max_iter=k) for k in (j - 1, j))
    assert (it0, it1) == (j - 1, j)
    assert r0 > 1.05 * r1
    tol = min(1.15 * r1, float(np.sqrt(r0 * r1)))
    it, res = solve(solver_tol=tol, gmres_restart=50)
    assert it == j
    assert res <= tol
