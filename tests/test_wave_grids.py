"""Wave-space mobility on every grid size with a specialised transform, and on grids that take the
generic passes (other sizes, Ny != Nz), against the FP64 oracle.

The box edge is chosen so that the set-up picks the wanted grid.  Tolerance: FP32 spreading, transforms
and contraction against FP64; a sum of n FP32 terms of random rounding is off by about sqrt(log2 n) eps
per transform pass, 1e-6 relative at the largest grid here, and 1e-5 leaves a factor of ten.
"""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from fsd_b200.core import FSD
from oracle import fsd_oracle as O

XI, ERR = 0.5, 1e-3
KMAX = int(2.0 * math.sqrt(-math.log(ERR)) * XI) + 1


def edge(n):
    return (n - 0.5) * math.pi / KMAX


CUBIC = [12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120,
         128, 135, 144, 150]
OTHER = [(125, 125, 125), (160, 24, 24), (16, 27, 27), (45, 12, 12), (30, 24, 27), (12, 160, 160), (125, 20, 20)]


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [(n, n, n) for n in CUBIC] + OTHER, ids=lambda g: "x".join(map(str, g)))
def test_wave_mobility_on_grid(cuda, grid):
    n = grid
    L = tuple(edge(k) for k in n)
    xy = 0.2 if n[0] % 2 == 0 else 0.0
    N = 12
    rng = np.random.default_rng(sum(n))
    frac = rng.random((N, 3)) - 0.5
    pos = np.zeros((N, 4), np.float32)
    pos[:, 1] = frac[:, 1] * L[1]
    pos[:, 2] = frac[:, 2] * L[2]
    pos[:, 0] = frac[:, 0] * L[0] + xy * pos[:, 1]
    s = FSD(N, (*L, xy), error=ERR, xi=XI, gmres_restart=2, lanczos_max=4)
    info = s.pse_info()
    assert (info.Nx, info.Ny, info.Nz) == n
    F = rng.standard_normal(11 * N).astype(np.float32)
    got = s.mobility(torch.as_tensor(pos).cuda().view(-1), torch.as_tensor(F).cuda(), parts=1).cpu().numpy()
    s.close()
    # the oracle on the set-up's own grid parameters (pinned by the set-up tests)
    gp = {k: getattr(info, k) for k in ("Nx", "Ny", "Nz", "P", "eta", "hx", "hy", "hz")}
    Ff, C = O.split_generalized(F.astype(np.float64), N)
    O.FFT_WORKERS = 8
    try:
        u, D = O.wave_space(pos, Ff, C, L, xy, gp, XI)
    finally:
        O.FFT_WORKERS = 1
    ref = O.generalized_velocity(u, np.transpose(D, (0, 2, 1)), N)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-5
