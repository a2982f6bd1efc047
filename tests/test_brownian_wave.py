"""The launches of the far-field Brownian slip."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from fsd_b200 import _lib
from fsd_b200.core import FSD

pytestmark = pytest.mark.gpu

XI, ERR = 0.5, 1e-3
KMAX = int(2.0 * math.sqrt(-math.log(ERR)) * XI) + 1


def system(N, grid, xy, **kw):
    L = tuple((n - 0.5) * math.pi / KMAX for n in grid)
    rng = np.random.default_rng(sum(grid) + N)
    sites = np.stack(np.unravel_index(rng.permutation(27)[:N], (3, 3, 3)), 1)  # no two spheres overlap
    frac = (sites + 0.5 + 0.1 * rng.random((N, 3))) / 3.0 - 0.5
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = frac * np.array(L)
    pos[:, 0] += xy * pos[:, 1]
    s = FSD(N, (*L, xy), error=ERR, xi=XI, gmres_restart=2, T=1.0, dt=1.0, seed=9, **kw)
    info = s.pse_info()
    assert (info.Nx, info.Ny, info.Nz) == grid
    p = torch.as_tensor(pos).cuda().view(-1)
    s.build_neighbor_list(p)
    return s, p, pos, L


@pytest.mark.parametrize("grid,wave", [((16, 16, 16), 5), ((15, 16, 18), 6)])
def test_farfield_launches(cuda, grid, wave):
    """Noise, inverse transform (two launches on half spectra, three on full grids), contraction and combination for
    the wave part, and no binning: nothing is spread.  Normals, norm, first vector, combination and sum, and five
    launches per Lanczos step for the real part."""
    s, p, _, _ = system(6, grid, 0.0)
    s.brownian_farfield(p, 0)
    before = _lib.lib().fsd_launch_count()
    s.brownian_farfield(p, 1)
    n = _lib.lib().fsd_launch_count() - before
    assert n == wave + 5 + 5 * s.solve_info()["lanczos_ff_iters"]
    s.close()
