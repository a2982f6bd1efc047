"""Clusters of close-packed spheres at the sizes where rows, sets and groups of lanes begin and end, against
the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import ewald_golden
from fsd_b200.core import FSD
from oracle import fsd_oracle as O

pytestmark = pytest.mark.gpu

EDGE = 40.0
L = (EDGE, EDGE, EDGE)


def packed(N, spacing, seed, jitter=0.004):
    """The N sites of a face-centred cubic lattice nearest the box corner, jittered and wrapped."""
    k = np.arange(-9, 10)
    g = np.array(np.meshgrid(k, k, k)).reshape(3, -1).T
    g = g[g.sum(1) % 2 == 0] * (spacing / np.sqrt(2.0))
    rng = np.random.default_rng(seed)
    x = g[np.argsort((g ** 2).sum(1), kind="stable")[:N]]
    x = x + jitter * (2.0 * rng.random(x.shape) - 1.0) + EDGE / 2
    pos = np.zeros((N, 4), np.float32)
    pos[rng.permutation(N), :3] = x - EDGE * np.floor(x / EDGE + 0.5)
    return pos


def dev(x):
    return torch.as_tensor(np.ascontiguousarray(x, np.float32)).cuda().view(-1)


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def solver(pos, xy=0.0, **kw):
    s = FSD(len(pos), (*L, xy), **kw)
    p = dev(pos)
    s.build_neighbor_list(p)
    return s, p


@pytest.mark.parametrize("N", [1, 2, 3, 13, 20, 40, 151])
def test_approximate_inverse_of_every_set_size(cuda, N):
    """Sets from one member to the cap of 32.  FP64 normal equations, blocks stored in FP32: 1e-7 expected."""
    pos = packed(N, 2.03, N)
    s, p = solver(pos, precond="learned", learned_inner=0)
    s.precond_build(p)
    A = O.pruned_rfu_sparse(pos, L, 0.0, *O.resistance_table()).tocsr()
    G = O.spai2(A, N)
    b = np.random.default_rng(N).standard_normal(17 * N)
    assert rel(s.precond_apply(dev(b)).cpu().numpy(), O.saddle_precond(b, G, N)) < 1e-5
    s.close()


@pytest.mark.parametrize("N", [1, 2, 5, 31, 33, 257, 700])
@pytest.mark.parametrize("xy", [0.0, -0.5])
def test_pair_sums_of_small_and_odd_sizes(cuda, N, xy):
    """Real-space mobility and the four lubrication products, with a strain of its own on every particle; the velocity
    also from an address that is a multiple of four bytes only.  FP32 pair sums: 1e-6 expected, 1e-5 allowed."""
    pos = packed(N, 2.03, N)
    s, p = solver(pos, xy)
    pr = O.Problem(pos, L, xy, table=ewald_golden())
    rng = np.random.default_rng(N + 1)
    F, U = rng.standard_normal(11 * N).astype(np.float32), rng.standard_normal(6 * N).astype(np.float32)
    assert rel(s.mobility(p, dev(F), parts=2).cpu(), pr.mobility(F, parts=2)) < 1e-5
    got = s.rfu(p, dev(U))
    if N == 1:
        assert not got.any()
    else:
        assert rel(got.cpu(), pr.rfu(U)) < 1e-5
    odd = torch.zeros(6 * N + 1, device="cuda")
    odd[1:] = dev(U)
    assert torch.equal(s.rfu(p, odd[1:]), got)
    sl = s.rsu(p, dev(U))
    assert torch.equal(s.rsu(p, odd[1:]), sl)
    ori = rng.standard_normal((N, 3))
    ori = (ori / np.linalg.norm(ori, axis=1, keepdims=True)).astype(np.float32)
    mask = rng.random(N).astype(np.float32)
    active = dict(ori=ori, b2mask=mask, B2=-0.5)
    args = (pr.L, xy, pr.rows, pr.tdist, pr.tvals)
    for got, ref in ((sl, O.rsu(pos, U, *args)),
                     (s.rfe(p, 0.7, dev(ori), dev(mask), -0.5), O.rfe(pos, 0.7, *args, **active)),
                     (s.rse(p, 0.7, dev(ori), dev(mask), -0.5), O.rse(pos, 0.7, *args, **active))):
        if N == 1:
            assert not got.any() and not ref.any()
        else:
            assert rel(got.cpu(), ref) < 1e-5
    s.close()


@pytest.mark.parametrize("N,edge,xy", [(1, 13.0, 0.0), (2, 14.0, 0.5), (33, 15.0, -0.5), (300, 16.0, 0.31),
                                       (1025, 27.0, 0.49), (700, 40.0, 0.0)])
def test_neighbor_rows_at_few_cells(cuda, N, edge, xy):
    """Rows against all pairs where the box has two, three or four cells per axis, and the sheared image of a
    cell reaches the next; pairs within rounding of the list radius are left out of the comparison."""
    rng = np.random.default_rng(N)
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = (rng.random((N, 3)) - 0.5) * edge
    pos[:, 0] += xy * pos[:, 1]
    box = (edge,) * 3
    s = FSD(N, (*box, xy))
    s.build_neighbor_list(dev(pos))
    r = s.pse_info().ewald_cut + 0.4
    rows = s.neighbor_list()
    lo, hi = O.neighbor_list(pos, box, xy, r - 1e-5), O.neighbor_list(pos, box, xy, r + 1e-5)
    for got, a, b in zip(rows, lo, hi):
        assert len(np.unique(got)) == len(got)
        assert set(a) <= set(got) <= set(b)
    s.close()


@pytest.mark.parametrize("precond,inner", [("none", 0), ("learned", 0), ("learned", 4)])
@pytest.mark.parametrize("N", [1, 2, 3, 6, 31])
def test_solve_of_unaligned_lengths(cuda, N, precond, inner):
    """17 N of every remainder by four (rows of the Krylov basis that begin off a 16-byte boundary), and systems
    smaller than the number of iterations allowed."""
    pos = packed(N, 2.3, N)
    s, p = solver(pos, precond=precond, solver_tol=1e-6, gmres_restart=60, learned_inner=inner)
    s.precond_build(p)
    pr = O.Problem(pos, L, 0.0, table=ewald_golden())
    rhs = np.random.default_rng(N).standard_normal(17 * N)
    x, it, res, st = s.saddle_solve(p, dev(rhs))
    assert res < 1e-5
    assert rel(x.cpu().numpy(), pr.solve(rhs)) < 1e-4
    s.close()


@pytest.mark.parametrize("N", [2, 3, 5, 33, 257])
def test_nearfield_sample_is_the_square_root(cuda, N):
    """R_FU^(1/2) of the library's own normals against the dense FP64 square root.  The iteration stops when the
    sample changes by less than 1e-5 of itself; on this well separated lattice the sum of the remaining changes
    stays below a hundred times that."""
    pos = packed(N, 2.4, N)
    s, p = solver(pos, T=1.0, dt=1.0, seed=11, lanczos_tol=1e-5, lanczos_max=100)
    pr = O.Problem(pos, L, 0.0, table=ewald_golden())
    R = np.stack([pr.rfu(e) for e in np.eye(6 * N)])
    w, V = np.linalg.eigh((R + R.T) / 2)
    psi = s.draw_normals(3, 4, 6 * N).cpu().numpy().astype(np.float64)
    ref = np.sqrt(2.0) * (V @ (np.sqrt(np.maximum(w, 0.0)) * (V.T @ psi)))
    assert rel(s.brownian_nearfield(p, 4).cpu().numpy(), ref) < 1e-3
    s.close()


@pytest.mark.parametrize("N", [1, 2, 15, 17, 33])
def test_products_with_user_blocks_of_any_row_length(cuda, N):
    """G once, on rows of no block to N blocks (N > 16 lanes of operand pairs, N > 32 of blocks).  FP32 rows of at
    most 6 N terms: 1e-6 expected."""
    s, p = solver(packed(N, 2.3, N), precond="learned", learned_inner=0)
    rng = np.random.default_rng(N)
    n = np.minimum(N, np.arange(N) * 2)
    n[-1] = N
    rowptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    col = np.concatenate([rng.permutation(N)[:k] for k in n]).astype(np.int32)
    blocks = rng.standard_normal((len(col), 6, 6)).astype(np.float32)
    s.precond_set_blocks(torch.as_tensor(rowptr).cuda(), torch.as_tensor(col).cuda(), torch.as_tensor(blocks).cuda())
    G = np.zeros((6 * N, 6 * N))
    for i in range(N):
        for e in range(rowptr[i], rowptr[i + 1]):
            G[6 * i:6 * i + 6, 6 * col[e]:6 * col[e] + 6] += blocks[e]
    b = rng.standard_normal(17 * N)
    s.precond_build(p)
    x = dev(b)
    got = s.precond_apply(x).cpu().numpy()
    assert rel(got, O.saddle_precond(b.astype(np.float32).astype(np.float64), G, N)) < 1e-5
    s.close()


@pytest.mark.parametrize("N", [8, 295, 2368, 2369, 3000])
def test_overlapped_launches_keep_their_order(cuda, N):
    """Chains of dependent launches on either side of the grid size up to which they overlap: the same bits in
    every repetition, interleaved with other products, and the pair sums against the oracle."""
    pos = packed(N, 2.2, N)
    s, p = solver(pos)
    rng = np.random.default_rng(N)
    F, U = rng.standard_normal(11 * N).astype(np.float32), dev(rng.standard_normal(6 * N))
    x = dev(rng.standard_normal(17 * N))
    Fd = dev(F)
    first = [s.mobility(p, Fd), s.rfu(p, U), s.saddle_multiply(p, x)]
    for _ in range(10):
        for a, b in zip(first, (s.mobility(p, Fd), s.rfu(p, U), s.saddle_multiply(p, x))):
            assert torch.equal(a, b)
    ref = O.Problem(pos, L, 0.0, table=ewald_golden()).mobility(F, parts=2)
    assert rel(s.mobility(p, Fd, parts=2).cpu(), ref) < 1e-5
    s.close()
