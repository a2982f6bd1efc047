"""Spreading and binning of the wave space where bins and tiles are uneven: every particle in one small
cluster (more members per tile than are staged at once, most tiles empty) across a box corner, stencils
wider than the smallest tiles, single particles, and the grids on either side of each tile shape's limit.

Tolerance as for the transforms on even bins: FP32 sums against FP64, 1e-6 expected, 1e-5 allowed.  A
cluster of m particles adds m random terms per node, whose rounding grows no faster than their sum.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import shutil
import subprocess
from pathlib import Path

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


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    """fsd_spread.h compiled on its own: spread_choice as (TX, TY, TZ, form, local), then the binning columns as
    (pieces of an axis, nodes per piece, columns)."""
    gxx, inc = shutil.which("g++"), Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    if gxx is None or not (inc / "cuda_runtime.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("spread")
    (d / "choice.cpp").write_text("""#include "fsd_spread.h"
extern "C" void choice(const int* grid, float xy, const int* tune, int* out) {
    fsd::GridParams g;
    g.Nx = grid[0], g.Ny = grid[1], g.Nz = grid[2], g.P = grid[3];
    TuneChoice t;
    t.TX = tune[0], t.TY = tune[1], t.TZ = tune[2], t.spread_rows = tune[3], t.set = tune[0] > 0;
    const fsd::SpreadChoice c = fsd::spread_choice(g, xy, t);
    out[0] = c.TX, out[1] = c.TY, out[2] = c.TZ, out[3] = c.form, out[4] = c.local;
    out[5] = fsd::bin_pieces(g.Nz), out[6] = fsd::bin_piece_nodes(g.Nz), out[7] = (int)fsd::bin_columns(g);
}
""")
    csrc = Path(__file__).resolve().parents[1] / "fsd_b200" / "csrc"
    subprocess.run([gxx, "-std=c++17", "-shared", "-fPIC", f"-I{csrc}", f"-I{inc}", "-o", str(d / "choice.so"),
                    str(d / "choice.cpp")], check=True)
    f = C.CDLL(str(d / "choice.so")).choice
    f.argtypes = [C.POINTER(C.c_int), C.c_float, C.POINTER(C.c_int), C.POINTER(C.c_int)]

    def call(grid, xy, tune=(0, 0, 0, 0), part=slice(5)):
        out = (C.c_int * 8)()
        f((C.c_int * 4)(*grid), xy, (C.c_int * 4)(*tune), out)
        return tuple(out)[part]

    return call


@pytest.mark.parametrize("tile", [(4, 4, 8), (8, 8, 8), (4, 8, 16), (4, 4, 32)])
def test_four_nodes_per_lane_only_on_local_tiles(choose, tile):
    """A tuned tile with four nodes per lane holds for the tilts at which its separations are tile-relative and
    gives way to the built-in choice at the others (the kernel does not take minimum images)."""
    kept = left = 0
    for n in range(12, 151):
        for P in (6, 8, 10):
            if n - P + 1 < max(tile):
                continue
            for xy in (0.0, 0.1, -0.3, 0.45, -0.5):
                got = choose((n, n, n, P), xy, (*tile, 2))
                if all((t + P) * (1 + abs(xy)) < 0.5 * n for t in tile):
                    assert got == (*tile, 2, 1)
                    kept += 1
                else:
                    assert got == choose((n, n, n, P), xy)
                    assert got[3] != 2 or got[4]
                    left += 1
    assert kept and left


def test_binning_columns_are_short(choose):
    """A warp's work on a column grows with the square of its length: at most 160 nodes, in pieces that cover the
    axis with none empty."""
    for nz in range(12, 4000):
        pieces, nodes, columns = choose((12, 16, nz, 6), 0.0, part=slice(5, 8))
        assert nodes <= 160 and (pieces - 1) * nodes < nz <= pieces * nodes
        assert columns == 12 * 16 * pieces
        assert pieces == 1 or nz > 160


@pytest.mark.gpu
@pytest.mark.parametrize("grid,N,size", [((12, 12, 162), 300, 1.0), ((15, 12, 432), 2000, 1.0), ((12, 12, 512), 900, 0.1),
                                         ((12, 16, 324), 1500, 1.0)])
def test_spread_on_axes_of_several_pieces(cuda, grid, N, size):
    """Particles spread over the box, and clustered around the middle of the long axis, where pieces meet, and its
    end, where they wrap.  Oracle and tolerance as for the other spreading tests, on axes short enough for it: the
    Green function's sin k - k cos k in FP32 cancels to 3 eps / k^2, 1e-3 of the factors of the lowest mode at 500
    nodes, which is 1e-5 of the product when particles fill the box."""
    L = tuple(edge(n, 1e-3) for n in grid)
    rng = np.random.default_rng(grid[2] + N)
    frac = rng.random((N, 3)) - 0.5
    frac[:, 2] = size * frac[:, 2] + (0.0 if size == 1.0 else np.where(np.arange(N) % 2, 0.5, 0.0))
    frac -= np.floor(frac + 0.5)
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = frac * np.array(L)
    s = FSD(N, (*L, 0.0), xi=XI, gmres_restart=2, lanczos_max=4)
    info = s.pse_info()
    assert (info.Nx, info.Ny, info.Nz) == grid
    F = torch.as_tensor(rng.standard_normal(11 * N).astype(np.float32)).cuda()
    p = torch.as_tensor(pos).cuda().view(-1)
    got = s.mobility(p, F, parts=1)
    assert torch.equal(s.mobility(p, F, parts=1), got)
    s.close()
    gp = {k: getattr(info, k) for k in ("Nx", "Ny", "Nz", "P", "eta", "hx", "hy", "hz")}
    Ff, Cp = O.split_generalized(F.cpu().numpy().astype(np.float64), N)
    u, D = O.wave_space(pos, Ff, Cp, L, 0.0, gp, XI)
    ref = O.generalized_velocity(u, np.transpose(D, (0, 2, 1)), N)
    assert np.linalg.norm(got.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("n,N", [(60, 4000), (60, 16000), (36, 3000), (32, 1500), (54, 30000)])
def test_tuned_spreading_at_another_tilt(cuda, n, N):
    """Tiles tuned without tilt, then a tilt at which a tuned tile's separations need not be tile-relative, on the
    tuned handle and on a second one that takes its choice from the cache.  Against a handle that was not tuned; the
    forms round separations of up to half the box (4e-6 at 60 nodes) in different places, 8e-7 of the product."""
    L = (edge(n, 1e-3),) * 3
    rng = np.random.default_rng(n * N)
    frac = rng.random((N, 3)) - 0.5
    F = torch.as_tensor(rng.standard_normal(11 * N).astype(np.float32)).cuda()

    def at(xy):
        pos = np.zeros((N, 4), np.float32)
        pos[:, 1:3] = frac[:, 1:] * L[0]
        pos[:, 0] = frac[:, 0] * L[0] + xy * pos[:, 1]
        return torch.as_tensor(pos).cuda().view(-1)

    def handle(xy, tune):
        return FSD(N, (*L, xy), xi=XI, gmres_restart=2, lanczos_max=4, autotune=tune)

    plain = handle(0.0, 0)
    tuned = handle(0.0, 1)
    tuned.mobility(at(0.0), F, parts=1)
    cached = handle(0.45, 1)
    for xy in (0.45, -0.3, 0.0):
        for s in (plain, tuned, cached):
            s.set_box(*L, xy)
        ref = plain.mobility(at(xy), F, parts=1)
        for s in (tuned, cached):
            assert (s.mobility(at(xy), F, parts=1) - ref).norm() < 2e-6 * ref.norm()
    for s in (plain, tuned, cached):
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("P,strain", [(10, 1.0), (11, 1.15), (12, 1.3)])
@pytest.mark.parametrize("grid", [(12, 12, 12), (30, 30, 12), (12, 30, 24), (27, 12, 20)])
def test_spread_on_grids_as_wide_as_the_stencil(cuda, grid, P, strain):
    """Axes with one to three nodes more than the stencil has, P - 1: tiles of 1 to 48 nodes, which are no whole
    warps.  The oracle and tolerance of the other spreading tests."""
    N = 301
    L = tuple(edge(n, 1e-3) for n in grid)
    rng = np.random.default_rng(sum(grid) + P)
    frac = rng.random((N, 3)) - 0.5
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = frac * np.array(L)
    s = FSD(N, (*L, 0.0), xi=XI, max_strain=strain, gmres_restart=2, lanczos_max=4)
    info = s.pse_info()
    assert (info.Nx, info.Ny, info.Nz, info.P) == (*grid, P)
    F = torch.as_tensor(rng.standard_normal(11 * N).astype(np.float32)).cuda()
    got = s.mobility(torch.as_tensor(pos).cuda().view(-1), F, parts=1).cpu().numpy()
    s.close()
    gp = {k: getattr(info, k) for k in ("Nx", "Ny", "Nz", "P", "eta", "hx", "hy", "hz")}
    Ff, Cp = O.split_generalized(F.cpu().numpy().astype(np.float64), N)
    u, D = O.wave_space(pos, Ff, Cp, L, 0.0, gp, XI)
    ref = O.generalized_velocity(u, np.transpose(D, (0, 2, 1)), N)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-5
