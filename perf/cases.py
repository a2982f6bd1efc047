"""The work whose speed is measured: calls that a user's program makes on one suspension of N unit
spheres, from a few hundred particles (a replica of a parameter study) to the largest configuration
of this repository (N = 131072).

Kinds of case (all through fsd_b200.core.FSD on device tensors):
  step         one full Brownian time step with shear (neighbour list, preconditioner build, pair
               forces, both Brownian terms, drift, main solve, Euler); every pass starts from the
               state's configuration at the next timestep number, so it draws fresh noise
  solve        the three-vector saddle solve on its own, from a zero guess
  mobility     the far-field mobility product (the operator a Krylov solver applies)
  lubrication  a new configuration's neighbour list and its four near-field products
  precond      a new configuration's preconditioner and one application of it
  brownian     the far- and near-field Brownian samples of one timestep

Configurations are seeded: random points whose overlaps are pushed apart on the GPU, so that at
volume fractions from about 0.4 most particles have near-contact neighbours (gaps of 1e-3 to 2e-3),
as in the benchmark's suspensions, and below that gaps are spread out.
"""
import math
from pathlib import Path

import numpy as np
import torch

from fsd_b200.core import FSD

ROOT = Path(__file__).resolve().parents[1]
DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # one replica of a parameter study: the smallest suspensions, all launches and latency
        {"name": "step_500", "kind": "step", "N": 500, "phi": 0.2, "xy": 0.0, "precond": "gmres"},
        # dense sheared squirmers with stresslet output, an odd particle count, a tilted box
        {"name": "step_3877_active", "kind": "step", "N": 3877, "phi": 0.45, "xy": 0.15, "precond": "gmres",
         "active": True},
        # the benchmarked step: N = 32768 at phi = 0.4
        {"name": "step_32768", "kind": "step", "N": 32768, "phi": 0.4, "xy": 0.0, "precond": "gmres"},
        # one solve with the default preconditioner (RCM + IC(0)) at the size of the quick validation run
        {"name": "solve_ichol_1000", "kind": "solve", "N": 1000, "phi": 0.2, "xy": 0.0, "precond": "ichol"},
        # one solve with the network's interval polynomial, a mid-sized dense suspension
        {"name": "solve_poly_8000", "kind": "solve", "N": 8000, "phi": 0.45, "xy": 0.0, "precond": "poly"},
        # mobility products: the smallest grid, a tilted one at higher accuracy (P = 8), the
        # benchmark's 72^3 and the largest configuration's 120^3
        {"name": "mobility_1000", "kind": "mobility", "N": 1000, "phi": 0.2, "xy": 0.0, "error": 1e-3},
        {"name": "mobility_7351_p8", "kind": "mobility", "N": 7351, "phi": 0.35, "xy": 0.25, "error": 1e-4},
        {"name": "mobility_32768", "kind": "mobility", "N": 32768, "phi": 0.4, "xy": 0.0, "error": 1e-3},
        {"name": "mobility_131072", "kind": "mobility", "N": 131072, "phi": 0.3, "xy": 0.0, "error": 1e-3},
        # near-field products of a new configuration
        {"name": "lubrication_32768", "kind": "lubrication", "N": 32768, "phi": 0.4, "xy": 0.1},
        # preconditioner of a new configuration and one application
        {"name": "precond_32768", "kind": "precond", "N": 32768, "phi": 0.4, "xy": 0.0, "precond": "gmres"},
        # Brownian samples of one timestep
        {"name": "brownian_20011", "kind": "brownian", "N": 20011, "phi": 0.3, "xy": 0.0},
    ]


def draw(rng):
    kind = rng.choice(["step", "solve", "mobility", "mobility", "lubrication", "precond", "brownian"])
    precond = rng.choice(["gmres", "poly", "ichol"]) if kind == "solve" else "gmres"
    top = {"step": 20000, "solve": 1500 if precond == "ichol" else 16000, "mobility": 120000}.get(kind, 32000)
    case = {
        "kind": kind,
        "N": int(round(math.exp(rng.uniform(math.log(500), math.log(top))))),
        "phi": round(rng.uniform(0.1, 0.25 if precond == "ichol" else 0.48 if kind == "mobility" else 0.42), 3),
        "xy": rng.choice([0.0, round(rng.uniform(-0.3, 0.3), 3)]),
    }
    if kind == "mobility":
        case["error"] = rng.choice([1e-3, 1e-3, 1e-4])
        if case["N"] > 40000:  # no dearer than the largest listed case
            case["error"], case["phi"] = 1e-3, max(case["phi"], 0.3)
    if kind in ("step", "solve", "precond"):
        case["precond"] = precond
    if kind == "step":
        case["active"] = rng.random() < 0.3
    return case


# ------------------------------------------------------------------ configurations
def _edge(N, phi):
    return (4.0 * math.pi * N / (3.0 * phi)) ** (1.0 / 3.0)


def _min_image(d, L, xy):
    img = torch.round(d[..., 2] / L)
    z = d[..., 2] - L * img
    img = torch.round(d[..., 1] / L)
    x = d[..., 0] - L * xy * img
    y = d[..., 1] - L * img
    return torch.stack([x - L * torch.round(x / L), y, z], -1)


def _candidates(pos, L, xy, r):
    """(N, C) candidate neighbours (-1: none) that hold everything within r of each particle, from cells
    of the (sheared) box; positions are unwrapped relative to any origin."""
    N = pos.shape[0]
    dev = pos.device
    nx = max(1, int(L / (math.sqrt(1.0 + xy * xy) * r)))
    ny = max(1, int(L / r))
    n = torch.tensor([nx, ny, ny], device=dev)
    f = torch.stack([pos[:, 0] - xy * pos[:, 1], pos[:, 1], pos[:, 2]], 1) / L
    f = f - torch.floor(f)
    c = torch.minimum((f * n).long(), n - 1)
    key = (c[:, 0] * ny + c[:, 1]) * ny + c[:, 2]
    order = torch.argsort(key, stable=True)
    ks = key[order]
    start = torch.searchsorted(ks, torch.arange(nx * ny * ny, device=dev))
    rank = torch.arange(N, device=dev) - start[ks]
    table = torch.full((nx * ny * ny, int(rank.max()) + 1), -1, dtype=torch.long, device=dev)
    table[ks, rank] = order
    o = torch.arange(-1, 2, device=dev)
    offs = torch.unique(torch.cat([torch.cartesian_prod(o, o, o) % n]), dim=0)
    nb = (c[:, None, :] + offs[None]) % n
    return table[(nb[..., 0] * ny + nb[..., 1]) * ny + nb[..., 2]].reshape(N, -1)


def _near(pos, L, xy, r, most):
    """(N, most) nearest neighbours within r, padded with the particle itself."""
    cand = _candidates(pos, L, xy, r)
    me = torch.arange(pos.shape[0], device=pos.device)[:, None]
    d = _min_image(pos[cand.clamp(min=0)] - pos[:, None], L, xy)
    r2 = d.square().sum(-1)
    r2 = torch.where((cand < 0) | (cand == me), torch.full_like(r2, 1e9), r2)
    v, i = torch.topk(r2, min(most, r2.shape[1]), dim=1, largest=False)
    return torch.where(v < r * r, torch.gather(cand, 1, i), me)


def suspension(N, phi, xy, seed):
    """Non-overlapping unit spheres (smallest gap 1e-3) in a cubic box with an xy tilt, centred on the
    origin: (N, 4) float32 on the GPU, and the edge."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    L = _edge(N, phi)
    pos = (torch.rand(N, 3, generator=g, dtype=F64) * L).to(DEV)
    # below phi = 0.38 each particle keeps a distance of its own, so that gaps spread out
    halo = max(0.0, (0.38 / phi) ** (1.0 / 3.0) - 1.0) * torch.rand(N, generator=g, dtype=F64).to(DEV)
    me = torch.arange(N, device=DEV)[:, None]
    for rounds in range(400):
        nb = _near(pos, L, xy, min(2.3 + float(halo.max()) * 2, L / 3.01), 24)
        want = 2.0 + 1.5e-3 + halo[:, None] + halo[nb]
        factor = 0.51 if rounds < 20 else 0.65
        if rounds == 60:  # a halo that does not fit is given up
            halo = torch.zeros_like(halo)
        for _ in range(10):
            d = _min_image(pos[nb] - pos[:, None], L, xy)
            r = d.square().sum(-1).sqrt().clamp(min=1e-9)
            push = torch.where((nb != me) & (r < want), (want - r) / r, torch.zeros_like(r))
            pos = pos - factor * (push[..., None] * d).sum(1)
        nb = _near(pos, L, xy, 2.05, 24)
        r = _min_image(pos[nb] - pos[:, None], L, xy).square().sum(-1).sqrt()
        if float(torch.where(nb != me, r, torch.full_like(r, 9.0)).min()) >= 2.0 + 1e-3:
            break
    # wrap into the box centred on the origin
    p = pos - L / 2.0
    k = torch.floor(p[:, 1] / L + 0.5)
    y = p[:, 1] - L * k
    x = p[:, 0] - xy * L * k
    x = x - L * torch.floor((x - xy * y) / L + 0.5)
    z = p[:, 2] - L * torch.floor(p[:, 2] / L + 0.5)
    out = torch.stack([x, y, z, torch.zeros_like(x)], 1).float()
    # float32 coordinates strictly inside the box
    out[:, 2] = torch.where(out[:, 2] >= L / 2, out[:, 2] - L, out[:, 2])
    return out.contiguous(), L


def prepare(case, seed):
    kind, N, xy = case["kind"], case["N"], case["xy"]
    pos, L = suspension(N, case["phi"], xy, seed)
    g = torch.Generator(device="cpu").manual_seed(seed + 1)

    def rand(*shape):
        return torch.randn(*shape, generator=g).to(DEV)

    opts = {}
    if kind in ("step", "solve", "precond"):
        form = case["precond"]
        opts = dict(solver_tol=1e-4, gmres_max_iter=3000, gmres_restart=100)
        if form == "ichol":
            opts.update(precond="ichol")
        else:
            opts.update(precond="learned", learned_inner=6 if form == "gmres" else 0,
                        learned_poly=10 if form == "poly" else 0)
    if kind in ("step", "brownian"):
        opts.update(T=1.0, dt=1e-4, lanczos_tol=1e-3, rfd_epsilon=1e-3)
    if case.get("active"):
        opts.update(sqm_B1=1.0, sqm_B2=-0.5, rot_diff=0.05, period=1)
    s = FSD(N, (L, L, L, xy), device=DEV, seed=seed % 65536, error=case.get("error", 1e-3), **opts)
    if opts.get("learned_poly"):
        s.learned_set_weights(np.fromfile(ROOT / "fsd_b200" / "data" / "learned_poly_k10.f32", "<f4"))
    st = {"case": case, "s": s, "pos": pos, "L": L, "t": 0}
    ori = rand(N, 3)
    st["ori"] = (ori / ori.norm(dim=1, keepdim=True)).contiguous()
    if kind == "step":
        st["image"] = torch.zeros(3 * N, dtype=torch.int32, device=DEV)
        st["force"] = torch.zeros(6 * N, device=DEV)
    elif kind == "mobility":
        st["F"] = rand(11 * N)
        s.build_neighbor_list(pos)
    elif kind == "lubrication":
        st["U"] = rand(6 * N)
    elif kind == "precond":
        st["b"] = rand(17 * N)
    elif kind == "brownian":
        s.build_neighbor_list(pos)
    elif kind == "solve":
        # the drift's right-hand side (0; -psi) plus an imposed shear on the stresslet rows
        rhs = torch.zeros(17 * N, device=DEV)
        rhs[11 * N:] = -rand(6 * N)
        rhs[6 * N + 1:11 * N:5] = 1.0
        st["rhs"] = rhs
        s.build_neighbor_list(pos)
        s.precond_build(pos)
    return st


def run(st):
    s, kind, pos = st["s"], st["case"]["kind"], st["pos"]
    if kind == "mobility":
        return s.mobility(pos, st["F"])
    if kind == "lubrication":
        s.build_neighbor_list(pos)
        return {"rfu": s.rfu(pos, st["U"]), "rfe": s.rfe(pos, 1.0, st["ori"], None, -0.5),
                "rsu": s.rsu(pos, st["U"]), "rse": s.rse(pos, 1.0, st["ori"], None, -0.5)}
    if kind == "precond":
        s.build_neighbor_list(pos)
        s.precond_build(pos)
        return s.precond_apply(st["b"])
    if kind == "solve":
        return s.saddle_solve(pos, st["rhs"])[0]
    if kind == "brownian":
        st["t"] += 1
        return {"slip": s.brownian_farfield(pos, st["t"]), "force": s.brownian_nearfield(pos, st["t"])}
    p, ori, image = pos.clone(), st["ori"].clone(), st["image"].clone()
    V = torch.empty(11 * s.N, device=DEV)
    s.step(st["t"], 1.0, p, ori, image, st["force"], V)
    st["t"] += 1
    return {"pos": p, "ori": ori, "image": image, "velocity": V}


# ------------------------------------------------------------------ work and tolerance
def _grid(case):
    """Nodes and stencil width of the wave-space grid (spacing pi / kmax, then the next 2-3-5 size)."""
    xi, err = 0.5, case.get("error", 1e-3)
    q = math.sqrt(-math.log(err))
    kmax = int(2.0 * q * xi) + 1
    n = int(kmax * _edge(case["N"], case["phi"]) / math.pi) + 1
    while True:
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1:
            return n ** 3, (6 if err >= 1e-3 else 8), q / xi
        n += 1


def work(case):
    """Bytes: particle inputs and outputs once.  Operations: what the operators' sums and transforms
    take (pairs counted within their cutoffs), for `solve` and `step` times the operator
    applications that a well-preconditioned solve to 1e-4 needs (20 each)."""
    kind, N, phi = case["kind"], case["N"], case["phi"]
    G, P, cut = _grid(case)
    density = 3.0 * phi / (4.0 * math.pi)
    real = density * 4.0 / 3.0 * math.pi * cut ** 3
    near = density * 4.0 / 3.0 * math.pi * 4.0 ** 3
    wave = 2 * N * P ** 3 * 2 * 11 + 2 * 11 * 2.5 * G * math.log2(G) + 200 * G
    mob = wave + N * real * 150
    rfu = N * near * 100
    inner = 7 * N * 12 * 72
    if kind == "mobility":
        return {"bytes": N * (16 + 44 + 44), "flops": mob}
    if kind == "lubrication":
        return {"bytes": N * (16 + 24 + 12 + 24 + 24 + 20 + 20), "flops": 4 * rfu}
    if kind == "precond":
        return {"bytes": N * (16 + 68 + 68), "flops": inner + N * 72 ** 3 / 3}
    if kind == "brownian":
        return {"bytes": N * (16 + 44 + 24), "flops": wave / 2 + 6 * N * real * 150 + 10 * rfu}
    solve = 20 * (mob + rfu + inner)
    if kind == "solve":
        return {"bytes": N * (16 + 68 + 68), "flops": solve}
    return {"bytes": N * (16 + 12 + 12 + 24 + 44 + 40), "flops": 3 * solve}


def tolerance(case):
    """Relative 2-norm, measured.  The operators are float32 sums: 1.3e-6 (mobility), 1.1e-7 (near field)
    and 2e-6 (preconditioner) off their 64-bit values.  The iterative paths stop at a relative residual of
    1e-4 (solves) or a relative change of 1e-3 (Brownian samples): sums in another order moved a step's
    velocity by 4e-5 and a solution by 3e-5, and a preconditioner with one more or fewer inner step, which
    moves the iteration at which a solve stops, by 2e-3 and 5e-4."""
    kind = case["kind"]
    if kind == "mobility":
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "lubrication":
        return {"rel": 2e-6, "max": 2e-4}
    if kind == "precond":
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "brownian":
        return {"rel": 2e-3, "max": 0.1}
    if kind == "solve":
        return {"rel": 2e-3, "max": 0.1}
    return {"rel": 8e-3, "max": 0.2, "differ": 1e-3}


# ------------------------------------------------------------------ 64-bit results
def exact(case, seed):
    """float64 torch restatements of the operators.  None for the paths whose result is where an
    iteration stopped (solves, Brownian samples, steps: a 64-bit solution of the same system differs by
    the solver's tolerance, and takes minutes), and for preconditioners too large for the dense
    arithmetic used here."""
    kind = case["kind"]
    if kind not in ("mobility", "lubrication", "precond") or (kind == "precond" and case["N"] > 3000):
        return None
    st = prepare(case, seed)
    if kind == "mobility":
        return _mobility64(st)
    if kind == "lubrication":
        return _lubrication64(st)
    return _precond64(st)


def _pairs(pos4, L, xy, cut):
    """Directed pairs closer than cut (with a margin); separations j - i rounded in float32 as the pair
    sums define them (the gap's float32 value is part of the result), as float64."""
    pos = pos4[:, :3]
    Lf = torch.tensor(L, dtype=torch.float32, device=DEV)
    xyf = torch.tensor(xy, dtype=torch.float32, device=DEV)
    inv = torch.tensor(1.0, dtype=torch.float32, device=DEV) / Lf
    out = []
    cand = _candidates(pos.double(), L, xy, min(cut + 0.01, L / 2))
    for a in range(0, pos.shape[0], 8192):
        c = cand[a:a + 8192]
        me = torch.arange(a, a + c.shape[0], device=DEV)[:, None].expand_as(c)
        d = pos[c.clamp(min=0)] - pos[me]
        img = torch.round(d[..., 2] * inv)
        z = d[..., 2] - Lf * img
        img = torch.round(d[..., 1] * inv)
        x = d[..., 0] - (Lf * xyf) * img
        y = d[..., 1] - Lf * img
        x = x - Lf * torch.round(x * inv)
        d2 = (x * x + y * y) + z * z
        ok = (c >= 0) & (c != me) & (d2 < cut * cut)
        out.append((me[ok], c[ok], torch.stack([x[ok], y[ok], z[ok]], 1), d2[ok].sqrt()))
    i, j, R, r = (torch.cat(v) for v in zip(*out))
    return i, j, R, r


def _couplet(genF, N):
    F6, S = genF[:6 * N].reshape(N, 6).double(), genF[6 * N:].reshape(N, 5).double()
    F, T = F6[:, :3], -F6[:, 3:]
    C = torch.zeros(N, 3, 3, dtype=F64, device=DEV)
    C[:, 0, 0], C[:, 1, 1], C[:, 2, 2] = S[:, 0], S[:, 4], -(S[:, 0] + S[:, 4])
    C[:, 0, 1], C[:, 1, 0] = S[:, 1] + 0.5 * T[:, 2], S[:, 1] - 0.5 * T[:, 2]
    C[:, 0, 2], C[:, 2, 0] = S[:, 2] - 0.5 * T[:, 1], S[:, 2] + 0.5 * T[:, 1]
    C[:, 1, 2], C[:, 2, 1] = S[:, 3] + 0.5 * T[:, 0], S[:, 3] - 0.5 * T[:, 0]
    return F, C


def _mobility64(st):
    s, pos4, L, xy, N = st["s"], st["pos"], st["L"], st["case"]["xy"], st["s"].N
    g, p = s.pse_info(), s.params
    xi, Lf, xyf = float(p.xi), float(p.Lx), float(p.xy)
    n, P = (g.Nx, g.Ny, g.Nz), g.P
    G = n[0] * n[1] * n[2]
    F, C = _couplet(st["F"], N)
    # stencil: first node from the float32 fractional coordinate
    f32 = torch.float32
    v = pos4[:, :3]
    Lt = torch.tensor(Lf, dtype=f32, device=DEV)
    d = v + Lt / 2
    d0 = (d[:, 0].double() - xyf * v[:, 1].double()).float()
    nt = torch.tensor(n, device=DEV)
    fr = torch.stack([d0, d[:, 1], d[:, 2]], 1) / Lt * nt.float()
    c = fr.long()
    first = c - P // 2 + 1 - (P % 2) * ((fr - c.float()) < 0.5).long()
    o = torch.arange(P, device=DEV)
    idx = (first[:, :, None] + o) % nt[:, None]  # N, 3, P
    h = [float(g.hx), float(g.hy), float(g.hz)]
    q = pos4[:, :3].double()
    eta = float(g.eta)
    expf = 2 * xi * xi / eta
    pref = (2 * xi * xi / 3.1415926536 / eta) ** 1.5
    spec = torch.zeros(12, G, dtype=F64, device=DEV)
    val = torch.cat([F, C.reshape(N, 9)], 1)  # N, 12
    chunk = max(1, 4_000_000 // P ** 3)

    def weights(a, b):
        ix, iy, iz = idx[a:b, 0], idx[a:b, 1], idx[a:b, 2]
        node = ((ix[:, :, None, None] * n[1] + iy[:, None, :, None]) * n[2] + iz[:, None, None, :])
        y = h[1] * iy.double() - Lf / 2
        x = h[0] * ix.double() - Lf / 2
        z = h[2] * iz.double() - Lf / 2
        dx = (x[:, :, None, None] + xyf * y[:, None, :, None]) - q[a:b, 0, None, None, None]
        dy = y[:, None, :, None] - q[a:b, 1, None, None, None]
        dz = z[:, None, None, :] - q[a:b, 2, None, None, None]
        dd = torch.stack(torch.broadcast_tensors(dx, dy, dz), -1)
        r = _min_image(dd, Lf, xyf)
        return node.reshape(b - a, -1), (pref * torch.exp(-expf * r.square().sum(-1))).reshape(b - a, -1)

    for a in range(0, N, chunk):
        b = min(N, a + chunk)
        node, w = weights(a, b)
        for k in range(12):
            spec[k].index_add_(0, node.reshape(-1), (w * val[a:b, k, None]).reshape(-1))
    spec = torch.fft.fftn(spec.reshape(12, *n), dim=(1, 2, 3))
    Fh, Ch = spec[:3], spec[3:].reshape(3, 3, *n)
    two_pi = 2.0 * 3.1416926536
    k = [torch.fft.fftfreq(m, 1.0 / m, dtype=F64, device=DEV) for m in n]
    k = [torch.where(t * 2 == -m, -t.abs(), t) for t, m in zip(k, n)]
    kx, ky, kz = torch.meshgrid(*k, indexing="ij")
    K = torch.stack([two_pi * kx / Lf, two_pi * (ky - xyf * kx) / Lf, two_pi * kz / Lf])
    k2 = K.square().sum(0)
    k2[0, 0, 0] = 1.0
    kk = k2.sqrt()
    w = 6.0 * 3.1415926536 * (1.0 + k2 / 4 / xi ** 2) * torch.exp(-(1 - eta) * k2 / 4 / xi ** 2) / k2 / G
    w[0, 0, 0] = 0.0
    j0 = torch.sin(kk) / kk
    j1 = (torch.sin(kk) - kk * torch.cos(kk)) / (k2 * kk)
    kdF = (K * Fh).sum(0) / k2
    Cdk = (Ch * K[None]).sum(1)
    kCk = (K * Cdk).sum(0) / k2
    U = torch.empty(12, *n, dtype=torch.complex128, device=DEV)
    for a in range(3):
        U[a] = (Fh[a] - K[a] * kdF) * (w * j0 * j0) + 1j * (Cdk[a] - K[a] * kCk) * (-w * j0 * 3 * j1)
        for b in range(3):
            U[3 + 3 * a + b] = 1j * (Fh[a] * K[b] - K[a] * K[b] * kdF) * (w * j0 * 3 * j1) + \
                (Cdk[a] * K[b] - K[a] * K[b] * kCk) * (9 * w * j1 * j1)
    del spec, Fh, Ch
    U = (torch.fft.ifftn(U, dim=(1, 2, 3)).real * G).reshape(12, G)
    quad = h[0] * h[1] * h[2]
    u = torch.zeros(N, 12, dtype=F64, device=DEV)
    for a in range(0, N, chunk):
        b = min(N, a + chunk)
        node, wt = weights(a, b)
        for t in range(12):
            u[a:b, t] = quad * (wt * U[t][node]).sum(1)
    del U
    # real space and self terms on the tabulated functions (fI, frr, g1, g2 | h1, h2, h3)
    tab = torch.as_tensor(s.ewald_table(), device=DEV).double().reshape(-1, 8)
    vel, D = u[:, :3].clone(), u[:, 3:].reshape(N, 3, 3).clone()
    i, j, R, r = _pairs(pos4, Lf, xyf, float(g.ewald_cut))
    i, j, R, r = (t[r >= g.ewald_dr] for t in (i, j, R, r))
    eye = torch.eye(3, dtype=F64, device=DEV)
    for a in range(0, len(i), 2_000_000):
        ii, jj, dist = i[a:a + 2_000_000], j[a:a + 2_000_000], r[a:a + 2_000_000].double()
        e = -R[a:a + 2_000_000].double() / dist[:, None]
        row = ((g.ewald_n * (dist - g.ewald_dr) / (g.ewald_cut - g.ewald_dr)).floor().long()).clamp(0, g.ewald_n - 1)
        fac = dist / g.ewald_dr - row - 1.0
        t = tab[row] + (tab[row + 1] - tab[row]) * fac[:, None]
        f1, f2, g1, g2, h1, h2, h3 = t[:, 0], t[:, 1], -t[:, 2], -t[:, 3], t[:, 4], t[:, 5], t[:, 6]
        Fj, Cj = F[jj], C[jj]
        eF = (e * Fj).sum(1)
        Ce, eC = (Cj * e[:, None, :]).sum(2), (Cj * e[:, :, None]).sum(1)
        eCe = (e * Ce).sum(1)
        col = lambda x: x[:, None]
        du = col(f1) * Fj + col((f2 - f1) * eF) * e + col(g1) * (Ce - col(eCe) * e) + col(g2) * (eC - col(4 * eCe) * e)
        ee = e[:, :, None] * e[:, None, :]
        m = lambda x: x[:, None, None]
        outer = lambda x, y: x[:, :, None] * y[:, None, :]
        dD = -m(g1) * (outer(Fj, e) - m(eF) * ee) - m(g2) * (m(eF) * eye + outer(e, Fj) - m(4 * eF) * ee)
        dD = dD + m(h1) * (Cj.transpose(1, 2) - 4 * Cj) + m(h2) * (outer(Ce, e) - m(eCe) * ee)
        dD = dD + m(h3) * (m(eCe) * eye + outer(e, Ce) + outer(eC, e) + outer(e, eC) - m(6 * eCe) * ee - Cj)
        vel.index_add_(0, ii, du)
        D.index_add_(0, ii, dD)
    vel += float(g.self_x) * F
    D += float(g.self_y) * (C.transpose(1, 2) - 4 * C)
    W = 0.5 * torch.stack([D[:, 2, 1] - D[:, 1, 2], D[:, 0, 2] - D[:, 2, 0], D[:, 1, 0] - D[:, 0, 1]], 1)
    E = torch.stack([2 * D[:, 0, 0] + D[:, 1, 1], D[:, 0, 1] + D[:, 1, 0], D[:, 0, 2] + D[:, 2, 0],
                     D[:, 1, 2] + D[:, 2, 1], 2 * D[:, 1, 1] + D[:, 0, 0]], 1)
    return torch.cat([torch.cat([vel, W], 1).reshape(-1), E.reshape(-1)])


def _resistance(dist32, first, count, precond=False):
    """Interpolated near-field scalars from the tabulated functions (1000 distances, 1000 x 22 values)."""
    raw = torch.from_numpy(np.fromfile(ROOT / "fsd_b200" / "data" / "resistance_table.bin", np.float32)).to(DEV)
    td, tv = raw[:1000].double(), raw[1000:].reshape(1000, 22)[:, first:first + count].double()
    r = dist32.double()
    small = float(np.float32(0.0001))
    ind = (torch.log10(((r - 2.0) / small).clamp(min=1e-30).float()) / float(np.float32(0.004305))).long()
    out = torch.zeros(len(r), count, dtype=F64, device=DEV)
    ok = (ind < 999) & (ind >= 0)
    k = ind.clamp(0, 998)
    fac = (r - td[k]) / (td[k + 1] - td[k])
    out[ok] = (tv[k] + (tv[k + 1] - tv[k]) * fac[:, None])[ok]
    near = r <= (2.0 + small if precond else 2.001)
    out[near] = tv[0 if precond else 232]
    return out


def _eps(r):
    m = torch.zeros(len(r), 3, 3, dtype=F64, device=DEV)
    m[:, 0, 1], m[:, 0, 2], m[:, 1, 2] = r[:, 2], -r[:, 1], r[:, 0]
    return m - m.transpose(1, 2)


def _lubrication64(st):
    s, N, xy = st["s"], st["s"].N, float(st["s"].params.xy)
    i, j, R, dist = _pairs(st["pos"], float(s.params.Lx), xy, 4.0)
    r = (R / dist[:, None]).double()
    U = st["U"].reshape(N, 6).double()
    b2 = 0.6 * -0.5
    o = st["ori"].double()
    e = torch.stack([b2 * (o[:, 0] ** 2 - o[:, 2] ** 2), 1.0 + b2 * 2 * o[:, 0] * o[:, 1], b2 * 2 * o[:, 0] * o[:, 2],
                     b2 * 2 * o[:, 1] * o[:, 2], b2 * (o[:, 1] ** 2 - o[:, 2] ** 2)], 1)
    E = torch.zeros(N, 3, 3, dtype=F64, device=DEV)
    E[:, 0, 0], E[:, 1, 1], E[:, 2, 2] = (2 * e[:, 0] - e[:, 4]) / 3, (2 * e[:, 4] - e[:, 0]) / 3, -(e[:, 0] + e[:, 4]) / 3
    E[:, 0, 1] = E[:, 1, 0] = 0.5 * e[:, 1]
    E[:, 0, 2] = E[:, 2, 0] = 0.5 * e[:, 2]
    E[:, 1, 2] = E[:, 2, 1] = 0.5 * e[:, 3]
    out = {k: torch.zeros(N, n, dtype=F64, device=DEV) for k, n in (("rfu", 6), ("rfe", 6), ("rsu", 5), ("rse", 5))}
    eye = torch.eye(3, dtype=F64, device=DEV)
    comp = lambda M: torch.stack([M[:, 0, 0], M[:, 0, 1], M[:, 0, 2], M[:, 1, 2], M[:, 1, 1]], 1)
    for a in range(0, len(i), 1_000_000):
        sl = slice(a, a + 1_000_000)
        ii, jj, rr, dd = i[sl], j[sl], r[sl], dist[sl]
        eps = _eps(rr)
        P = rr[:, :, None] * rr[:, None, :]
        Q = eye - P
        dot = lambda M, v: (M * v[:, None, :]).sum(2)
        ui, wi, uj, wj = U[ii, :3], U[ii, 3:], U[jj, :3], U[jj, 3:]
        XA, XB, YA, YB, YB11, YB12, XC, XD, YC, YD = _resistance(dd, 0, 10).T
        c = lambda x: x[:, None]
        F = c(XA) * dot(P, ui) + c(YA) * dot(Q, ui) + c(XB) * dot(P, uj) + c(YB) * dot(Q, uj)
        F = F - c(YB11) * dot(eps, wi) + c(YB12) * dot(eps, wj)
        T = c(YB11) * dot(eps, ui) + c(YB12) * dot(eps, uj) + c(XC) * dot(P, wi) + c(YC) * dot(Q, wi)
        T = T + c(XD) * dot(P, wj) + c(YD) * dot(Q, wj)
        out["rfu"].index_add_(0, ii, torch.cat([F, T], 1))
        XG11, XG12, YG11, YG12, YH11, YH12 = _resistance(dd, 10, 6).T
        Ei, Ej = dot(E[ii], rr), dot(E[jj], rr)
        rEi, rEj = (rr * Ei).sum(1), (rr * Ej).sum(1)
        F = -c((XG11 - 2 * YG11) * rEi) * rr - c(2 * YG11) * Ei + c((XG12 - 2 * YG12) * rEj) * rr + c(2 * YG12) * Ej
        T = c(2 * YH11) * dot(eps, Ei) + c(2 * YH12) * dot(eps, Ej)
        out["rfe"].index_add_(0, ii, torch.cat([F, T], 1))
        sym = lambda x, y: x[:, :, None] * y[:, None, :] + y[:, :, None] * x[:, None, :]
        m = lambda x: x[:, None, None]
        rui, ruj = (rr * ui).sum(1), (rr * uj).sum(1)
        S = m(XG11 * rui + XG12 * ruj) * (P - eye / 3)
        S = S + m(YG11) * (sym(ui, rr) - m(2 * rui) * P) + m(YG12) * (sym(uj, rr) - m(2 * ruj) * P)
        S = S + m(YH11) * sym(rr, dot(eps, wi)) + m(YH12) * sym(rr, dot(eps, wj))
        out["rsu"].index_add_(0, ii, -comp(S))
        XM11, XM12, YM11, YM12, ZM11, ZM12 = _resistance(dd, 16, 6).T
        S = 1.5 * m(XM11 * rEi + XM12 * rEj) * (P - eye / 3)
        S = S + m(0.5 * YM11) * (2 * sym(rr, Ei) - m(4 * rEi) * P) + m(0.5 * YM12) * (2 * sym(rr, Ej) - m(4 * rEj) * P)
        S = S + m(0.5 * ZM11) * (2 * E[ii] + (eye + P) * m(rEi) - 2 * sym(rr, Ei))
        S = S + m(0.5 * ZM12) * (2 * E[jj] + (eye + P) * m(rEj) - 2 * sym(rr, Ej))
        out["rse"].index_add_(0, ii, comp(S))
    return {k: v.reshape(-1) for k, v in out.items()}


def _precond64(st):
    """Inner GMRES on the pruned lubrication block, right-preconditioned by its two-hop sparse
    approximate inverse, between the saddle preconditioner's first and last steps."""
    s, N, xy = st["s"], st["s"].N, float(st["s"].params.xy)
    i, j, R, dist = _pairs(st["pos"], float(s.params.Lx), xy, float(s.params.rp))
    r = R.double() / dist.double()[:, None]
    c = _resistance(dist, 0, 10, precond=True)[:, :, None, None]
    P = r[:, :, None] * r[:, None, :]
    Q, eps = torch.eye(3, dtype=F64, device=DEV) - P, _eps(r)
    join = lambda a, b, d, e: torch.cat([torch.cat([a, b], 2), torch.cat([d, e], 2)], 1)
    off = join(c[:, 1] * P + c[:, 3] * Q, c[:, 5] * eps, c[:, 5] * eps, c[:, 7] * P + c[:, 9] * Q)
    own = join(c[:, 0] * P + c[:, 2] * Q, -c[:, 4] * eps, c[:, 4] * eps, c[:, 6] * P + c[:, 8] * Q)
    A = torch.zeros(N, 6, N, 6, dtype=F64, device=DEV)
    A[i, :, j, :] = off
    diag = torch.zeros(N, 6, 6, dtype=F64, device=DEV).index_add_(0, i, own)
    diag += torch.diag(torch.tensor([1.0] * 3 + [float(np.float32(1.33333333))] * 3, dtype=F64, device=DEV))
    me = torch.arange(N, device=DEV)
    A[me, :, me, :] = diag
    A = A.reshape(6 * N, 6 * N)
    # two-hop sets: the particle, its neighbours in index order, new members of their lists; at most 32
    rows = [[] for _ in range(N)]
    for a, b in sorted(zip(i.tolist(), j.tolist())):
        rows[a].append(b)
    cap = 32
    full = [sorted(v + [k]) for k, v in enumerate(rows)]
    sets = []
    for k in range(N):
        S = [k] + rows[k][:cap - 1]
        seen = set(S)
        for q in list(S[1:]):
            for t in full[q]:
                if t not in seen and len(S) < cap:
                    S.append(t)
                    seen.add(t)
        sets.append(S)
    size = max(len(S) for S in sets)
    idx = torch.tensor([S + [-1] * (size - len(S)) for S in sets], device=DEV)
    pad = (idx < 0)
    dof = (idx.clamp(min=0)[:, :, None] * 6 + torch.arange(6, device=DEV)).reshape(N, -1)
    pad6 = pad[:, :, None].expand(-1, -1, 6).reshape(N, -1)
    A2 = A @ A
    Gm = torch.zeros(N, 6, N, 6, dtype=F64, device=DEV)
    member = torch.zeros(N, N, dtype=torch.bool, device=DEV)
    member[me[:, None].expand_as(idx)[~pad], idx[~pad]] = True
    for a in range(0, N, 512):
        d, p6, ix, pd = dof[a:a + 512], pad6[a:a + 512], idx[a:a + 512], pad[a:a + 512]
        H = A2[d[:, :, None], d[:, None, :]]
        H = torch.where(p6[:, :, None] | p6[:, None, :], torch.zeros_like(H), H)
        H = H + torch.diag_embed(p6.double())
        k = me[a:a + 512]
        col = (k[:, None] * 6 + torch.arange(6, device=DEV))
        rhs = torch.where(p6[:, :, None], torch.zeros((), dtype=F64, device=DEV), A[d[:, :, None], col[:, None, :]])
        X = torch.linalg.solve(H, rhs).reshape(len(k), -1, 6, 6)
        keep = ~pd & member[ix.clamp(min=0), k[:, None]]
        kk = k[:, None].expand_as(ix)
        Gm[ix[keep], :, kk[keep], :] = X[keep]
    Gm = Gm.reshape(6 * N, 6 * N)
    b = st["b"].double()
    t = b[:6 * N] - b[11 * N:]
    steps = 6
    V, Z = [t / t.norm()], []
    H = torch.zeros(steps + 1, steps, dtype=F64, device=DEV)
    for q in range(steps):
        Z.append(Gm @ V[q])
        w = A @ Z[q]
        for _ in range(2):
            for a in range(q + 1):
                h = V[a] @ w
                H[a, q] += h
                w = w - h * V[a]
        H[q + 1, q] = w.norm()
        V.append(w / H[q + 1, q])
    rhs = torch.zeros(steps + 1, 1, dtype=F64, device=DEV)
    rhs[0] = t.norm()
    y = torch.stack(Z, 1) @ torch.linalg.lstsq(H, rhs).solution[:, 0]
    return torch.cat([b[:6 * N] - y, b[6 * N:11 * N], y])
