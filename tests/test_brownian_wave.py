"""The far-field Brownian slip part by part: its random field on half spectra and on full grids against FP64, and the
launches it takes."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from conftest import ewald_golden
from fsd_b200 import _lib
from fsd_b200.core import FSD
from oracle import fsd_oracle as O

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


def wave_slip(s, pos, L, xy, step):
    """The wave-space slip of the library's own normals in FP64: a conjugate-symmetric field drawn once per pair
    {k, -k} (at the pair's smaller index), mapped per Brownian_FarField.cu:113-374 and transformed as complex numbers."""
    g = {k: getattr(s.pse_info(), k) for k in ("Nx", "Ny", "Nz", "P", "eta", "hx", "hy", "hz")}
    n = (g["Nx"], g["Ny"], g["Nz"])
    h = (g["hx"], g["hy"], g["hz"])
    G = math.prod(n)
    z = s.draw_normals(2, step, 8 * G).cpu().numpy().astype(np.float64).reshape(G, 8)
    idx = np.arange(G)
    i, j, k = np.unravel_index(idx, n)
    m = np.ravel_multi_index(((n[0] - i) % n[0], (n[1] - j) % n[1], (n[2] - k) % n[2]), n)
    quad = math.prod(h)
    fac = math.sqrt(1.0 / quad)
    own = np.where((m == idx)[:, None], math.sqrt(2.0) * z[:, :3] + 0j, z[:, :3] + 1j * z[:, 3:6])
    f = fac * np.where((idx <= m)[:, None], own, np.conj(own[m])).T.reshape(3, *n)
    kx, ky, kz, w = O.gridk(n, L, xy, XI, g["eta"])
    kv = np.stack([kx, ky, kz])
    k2 = (kv ** 2).sum(0)
    k2[0, 0, 0] = 1.0
    kk = np.sqrt(k2)
    W = (f - kv * (kv * f).sum(0) / k2) * np.sqrt(w)
    W[:, 0, 0, 0] = 0.0
    U = np.fft.ifftn(np.sin(kk) / kk * W, axes=(1, 2, 3)).real * G
    D = np.fft.ifftn(1j * 3.0 * (np.sin(kk) - kk * np.cos(kk)) / (k2 * kk) * W[:, None] * kv[None], axes=(2, 3, 4)).real * G
    node = O.stencil(pos, L, xy, n, g["P"])
    r = O.min_image(O.node_positions(node, L, xy, h) - O.xyz(pos)[:, None, :], L, xy)
    x2 = 2.0 * XI * XI
    wgt = quad * (x2 / O.PI_REF / g["eta"]) ** 1.5 * np.exp(-x2 / g["eta"] * (r ** 2).sum(-1))
    flat = np.ravel_multi_index(np.moveaxis(node, -1, 0), n)
    u = np.einsum("np,cnp->nc", wgt, U.reshape(3, G)[:, flat])
    d = np.einsum("np,abnp->nab", wgt, D.reshape(3, 3, G)[:, :, flat])
    return O.generalized_velocity(u, np.transpose(d, (0, 2, 1)), len(pos))


@pytest.mark.parametrize("grid,xy", [((16, 16, 16), 0.0), ((15, 15, 15), 0.2), ((15, 16, 16), -0.3), ((16, 15, 15), 0.1),
                                     ((16, 15, 18), 0.2), ((15, 18, 16), 0.0), ((125, 15, 15), 0.0)],
                         ids=lambda g: "x".join(map(str, g)) if isinstance(g, tuple) else str(g))
def test_farfield_sample_of_the_librarys_normals(cuda, grid, xy):
    """Even and odd half spectra (the first four) and full grids (the others), each with the real-space part from the
    dense square root.  The Lanczos iteration stops at a relative change of 1e-6; 1e-4 leaves its remaining changes
    and FP32 a factor of ten."""
    N = 6
    s, p, pos, L = system(N, grid, xy, lanczos_tol=1e-6, lanczos_max=60)
    pr = O.Problem(pos, L, xy, table=ewald_golden())
    M = np.stack([pr.mobility(e, parts=2) for e in np.eye(11 * N)])
    w, V = np.linalg.eigh((M + M.T) / 2)
    psi = s.draw_normals(1, 3, 11 * N).cpu().numpy().astype(np.float64)
    real = math.sqrt(2.0) * (V @ (np.sqrt(np.maximum(w, 0.0)) * (V.T @ psi)))
    wave = wave_slip(s, pos, L, xy, 3)
    got = s.brownian_farfield(p, 3).cpu().numpy().astype(np.float64)
    s.close()
    assert np.linalg.norm(wave) > 0.05 * np.linalg.norm(real)
    assert np.linalg.norm(got - real - wave) < 1e-4 * np.linalg.norm(wave)


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
