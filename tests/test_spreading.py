"""Spreading and binning of the wave space where bins and tiles are uneven: every particle in one small
cluster (more members per tile than are staged at once, most tiles empty) across a box corner, stencils
wider than the smallest tiles, single particles, and the grids on either side of each tile shape's limit.

Tolerance as for the transforms on even bins: FP32 sums against FP64, 1e-6 expected, 1e-5 allowed.  A
cluster of m particles adds m random terms per node, whose rounding grows no faster than their sum.
"""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from fsd_b200.core import FSD
from oracle import fsd_oracle as O

XI = 0.5


def edge(n, err):
    return (n - 0.5) * math.pi / (int(2.0 * math.sqrt(-math.log(err)) * XI) + 1)


# grid, particles, cluster edge over box edge, shear strain, Ewald error
CASES = [(72, 700, 0.05, 0.2, 1e-3), (72, 1, 1.0, -0.3, 1e-3), (64, 333, 0.1, 0.0, 1e-4), (60, 257, 1.0, 0.45, 1e-3),
         (48, 900, 0.08, -0.5, 1e-4), (36, 129, 0.3, 0.1, 1e-5), (24, 400, 1.0, 0.3, 1e-3), (16, 65, 0.5, 0.2, 1e-4),
         (20, 31, 1.0, -0.2, 1e-5), (12, 200, 0.2, 0.0, 1e-3)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,N,size,xy,err", CASES)
def test_spread_uneven_bins(cuda, n, N, size, xy, err):
    L = (edge(n, err),) * 3
    rng = np.random.default_rng(n * N)
    frac = 0.5 + size * (rng.random((N, 3)) - 0.5)  # around the corner
    frac -= np.floor(frac + 0.5)
    pos = np.zeros((N, 4), np.float32)
    pos[:, 1:3] = frac[:, 1:] * L[0]
    pos[:, 0] = frac[:, 0] * L[0] + xy * pos[:, 1]
    s = FSD(N, (*L, xy), error=err, xi=XI, gmres_restart=2, lanczos_max=4)
    info = s.pse_info()
    F = torch.as_tensor(rng.standard_normal(11 * N).astype(np.float32)).cuda()
    p = torch.as_tensor(pos).cuda().view(-1)
    got = s.mobility(p, F, parts=1)
    again = s.mobility(p, F, parts=1)
    s.close()
    assert torch.equal(got, again)  # one writer per node, members in a fixed order
    gp = {k: getattr(info, k) for k in ("Nx", "Ny", "Nz", "P", "eta", "hx", "hy", "hz")}
    Ff, C = O.split_generalized(F.cpu().numpy().astype(np.float64), N)
    u, D = O.wave_space(pos, Ff, C, L, xy, gp, XI)
    ref = O.generalized_velocity(u, np.transpose(D, (0, 2, 1)), N)
    got = got.cpu().numpy()
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-5
