"""Device memory of the learned preconditioner: G once, the polynomial's copy of A by the blocks it has, and nothing
left to allocate when it is first applied."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsd_b200.core import FSD

pytestmark = pytest.mark.gpu

N, EDGE, CAP = 12000, 60.0, 32
MB = 1 << 20


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def lattice():
    """A face-centred cubic cluster: 13 blocks per row of A, at most 32 (the cap) per row of G."""
    k = np.arange(-24, 25)
    g = np.array(np.meshgrid(k, k, k)).reshape(3, -1).T
    g = g[g.sum(1) % 2 == 0] * (2.03 / np.sqrt(2.0))
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = g[np.argsort((g ** 2).sum(1), kind="stable")[:N]]
    assert np.abs(pos).max() < EDGE / 2
    return torch.as_tensor(pos).cuda().view(-1)


@pytest.mark.parametrize("form", [dict(learned_inner=4), dict(learned_inner=0), dict(learned_poly=6)],
                         ids=["inner", "once", "poly"])
def test_blocks_are_held_once(cuda, lattice, form):
    b = torch.ones(17 * N, device="cuda")
    for first in (True, False):  # the first handle also loads the kernels
        s = FSD(N, (EDGE, EDGE, EDGE, 0.0), precond="learned", lanczos_max=4, gmres_restart=4, **form)
        s.build_neighbor_list(lattice)
        f0 = free()
        s.precond_build(lattice)
        f1 = free()
        s.precond_apply(b)
        f2 = free()
        s.close()
    room = 9 / 8  # for growth
    blocks = 144 * N * (CAP * room + (13 * room if "learned_poly" in form else 0))
    work = 4 * N * (6 * 17 + 3 * CAP)  # basis, sets and lists
    # fifteen allocations round up to 2 MB; the result of the application and the graph's nodes are small
    assert f0 - f1 < blocks + work + 30 * MB
    assert f1 - f2 < 8 * MB
