"""The calls that a program solving the Poisson-Boltzmann boundary integral equation makes, at the sizes and
options that this repository's benchmark, golden cases and tests use, as timed cases.

A case is one call, or one short run of calls, of ``fabipb_b200.lib.Surface`` (or of the autograd function on it) on a
seeded closed surface of flat triangles.  ``kind`` says which:

  matvec    y = (D - K) x, the product that GMRES makes in each step; ``adjoint`` takes the transposed operator,
            ``direct`` the context that sums every panel pair, ``q`` the panel quadrature order
  solve     GMRES on a prepared context, preconditioner and right-hand side
  walks     the right-hand side and the solvation energy by the charge-tree walks
  gradient  the energy and its derivatives with respect to the charges, through torch.autograd
  program   everything a first run does: context, charges, preconditioner, right-hand side, GMRES, energy

Surfaces: ``sphere`` (icosphere), ``star`` (an octahedral geodesic sphere of 8 f^2 triangles, radially perturbed),
``shell`` (two such spheres, the inner one facing the cavity).  ``drop`` faces are left out, as the loader's filter of
sliver faces leaves them out of measured meshes, so that panel counts are odd too.  The panels are handed over in octree
order: vectors in the library's order and in the mesh's order are then the same thing.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cuda-fabipb_b200"))

from fabipb_b200 import lib, meshgen  # noqa: E402
from fabipb_b200.autograd import SolvationEnergy  # noqa: E402
from fabipb_b200.meshio import ChargeSet, PanelSet  # noqa: E402

KAPPA, EPS2 = 0.1257, 80.0
KCAL = 2.0 * math.pi * 332.0716
F64 = torch.float64
DENSE_MAX = 20500   # panels up to which exact() assembles the whole matrix (27 GB at most while it does)


def _case(name, kind, mesh, size, order, depth, mac, eps1, precision, **more):
    c = {"kind": kind, "mesh": mesh, "size": size, "drop": 0, "radius": 25.0, "order": order, "depth": depth, "mac": mac,
         "eps1": eps1, "precision": precision, "q": 1, "adjoint": False, "direct": False, "charges": 0, "precond": -1,
         "tol": 0.0}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest golden case: a coarse sphere, where launches and latency are all there is
        _case("matvec-sphere320-mixed", "matvec", "sphere", 2, 3, 2, 0.8, 1.0, "mixed", radius=20.0),
        # the Kirkwood sphere, the usual check of a set-up
        _case("matvec-sphere20480-mixed", "matvec", "sphere", 5, 3, 3, 0.8, 1.0, "mixed", radius=20.0),
        # a protein-sized surface with small leaves, in both precisions
        _case("matvec-star204800-mixed", "matvec", "star", 160, 4, 5, 0.7, 2.0, "mixed"),
        _case("matvec-star204800-fp64", "matvec", "star", 160, 4, 5, 0.7, 2.0, "fp64"),
        # the benchmark's capsid-scale surface: two shells, large leaves
        _case("matvec-shell2096704-mixed", "matvec", "shell", 362, 5, 5, 0.6, 2.0, "mixed", radius=230.0),
        # the transposed product of the adjoint solve, at a quarter of that surface, an odd number of panels
        _case("adjoint-shell524171-mixed", "matvec", "shell", 181, 5, 4, 0.6, 2.0, "mixed", radius=115.0, drop=5,
              adjoint=True),
        # the direct operator that FMM results are checked against
        _case("direct-star12797-fp64", "matvec", "star", 40, 4, 3, 0.7, 2.0, "fp64", drop=3, direct=True),
        # panel quadrature of order 2, where the one-point rule is too coarse
        _case("quad2-star2048-fp64", "matvec", "star", 16, 4, 3, 0.7, 2.0, "fp64", q=2),
        # many solves on a small prepared surface (titration states, poses)
        _case("solve-sphere1280-fp64", "solve", "sphere", 3, 3, 3, 0.8, 1.0, "fp64", radius=20.0, charges=100, precond=2,
              tol=1e-4),
        # right-hand side and energy of a protein's 20,000 charges on a prepared surface
        _case("walks-star204800-mixed", "walks", "star", 160, 4, 5, 0.7, 2.0, "mixed", charges=20000),
        # forces on the charges of a middle-sized surface
        _case("gradient-star19999-mixed", "gradient", "star", 50, 4, 4, 0.7, 2.0, "mixed", drop=1, charges=2000, precond=2,
              tol=1e-5),
        # a whole first run, from panels to the energy
        _case("program-star204800-mixed", "program", "star", 160, 4, 5, 0.7, 2.0, "mixed", charges=20000, precond=2,
              tol=1e-5),
    ]


def _depth(panels, surfaces, leaf):
    """The octree depth whose mean leaf is nearest `leaf` panels (about 4.4 * 4^depth leaves for each surface)."""
    return max(2, round(math.log(max(panels / (4.4 * surfaces * leaf), 1.0), 4)))


def draw(rng):
    kind = rng.choice(["matvec"] * 6 + ["solve", "solve", "walks", "gradient", "program", "program"])
    mesh = rng.choice(["star", "star", "shell"]) if kind in ("matvec", "walks") else "star"
    precision = rng.choice(["mixed", "mixed", "fp64"])
    surfaces = 2 if mesh == "shell" else 1
    direct = kind == "matvec" and rng.random() < 0.15
    q = 2 if kind == "matvec" and not direct and rng.random() < 0.12 else 1
    lo, hi = {"matvec": (300, 700000), "solve": (600, 60000), "walks": (3000, 300000), "gradient": (1000, 30000),
              "program": (5000, 100000)}[kind]
    if direct:
        lo, hi = 300, 20000
    if q == 2:
        lo, hi = 300, 6000
    panels = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    freq = max(5, round(math.sqrt(panels / (8.0 * surfaces))))
    leaf = math.exp(rng.uniform(math.log(30), math.log(250 if kind in ("matvec", "walks") else 50)))
    depth = _depth(panels, surfaces, leaf)
    order = rng.choice([3, 4, 5])
    radius = max(25.0, 25.0 * math.sqrt(panels / 2.0e5)) if surfaces == 1 else max(60.0, 230.0 * math.sqrt(panels / 2.1e6))
    return _case(None, kind, mesh, freq, order, depth, {3: 0.8, 4: 0.7, 5: 0.6}[order], rng.choice([1.0, 2.0]), precision,
                 drop=rng.randrange(0, 8), radius=round(radius, 3), q=q,
                 adjoint=kind == "matvec" and rng.random() < 0.25, direct=direct,
                 charges=0 if kind == "matvec" else max(20, round(panels / rng.uniform(8, 30))),
                 precond=2 if kind in ("solve", "gradient", "program") else -1,
                 tol=rng.choice([1e-4, 1e-5]) if kind in ("solve", "gradient", "program") else 0.0)


# ---------------------------------------------------------------------------------------------------------------------
# surfaces and charges
# ---------------------------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _unit_sphere(mesh, size):
    """Corners (F, 3, 3) of the unit sphere's triangles, counter-clockwise from outside; corners that faces share are the
    same numbers."""
    if mesh == "sphere":
        pos, faces = meshgen.icosphere(size)
        return torch.from_numpy(pos[faces]).cuda()
    i, j = (v.reshape(-1) for v in torch.meshgrid(torch.arange(size), torch.arange(size), indexing="ij"))
    up, down = i + j < size, i + j + 1 < size
    a, b = torch.stack([i, j], 1)[up], torch.stack([i, j], 1)[down]
    d = torch.tensor
    ij = torch.cat([torch.stack([a, a + d([1, 0]), a + d([0, 1])], 1),
                    torch.stack([b + d([1, 0]), b + d([1, 1]), b + d([0, 1])], 1)]).cuda()
    one = torch.cat([ij, size - ij.sum(2, keepdim=True)], 2)   # whole coordinates of one octant's corners
    faces = []
    for s in range(8):
        sign = d([1 - 2 * (s & 1), 1 - (s & 2), 1 - (s & 4) // 2]).cuda()
        f = one * sign
        faces.append(f if int(sign.prod()) > 0 else f[:, [0, 2, 1]])
    p = torch.cat(faces).to(F64)
    r = torch.sqrt(p[..., 0] * p[..., 0] + p[..., 1] * p[..., 1] + p[..., 2] * p[..., 2])
    return p / r[..., None]


class _Radius:
    """r(u) = R (1 + smooth seeded waves) on the unit sphere, and the surface's normals."""

    def __init__(self, radius, amplitude, rng):
        k = 10
        self.radius = radius
        self.w = rng.normal(size=(k, 3))
        self.w *= (rng.uniform(2.0, 6.0, k) / np.linalg.norm(self.w, axis=1))[:, None]
        self.a = amplitude * rng.normal(size=k) / math.sqrt(k)
        self.p = rng.uniform(0.0, 2.0 * math.pi, k)

    def __call__(self, u, normal=False):
        x, y, z = u[..., 0], u[..., 1], u[..., 2]
        f = torch.ones_like(x)
        g = [torch.zeros_like(x) for _ in range(3)]
        for (w0, w1, w2), a, p in zip(self.w.tolist(), self.a.tolist(), self.p.tolist()):
            t = w0 * x + w1 * y + w2 * z + p
            f += a * torch.cos(t)
            if normal:
                s = -a * torch.sin(t)
                for c, wc in enumerate((w0, w1, w2)):
                    g[c] += wc * s
        if not normal:
            return self.radius * f
        g = torch.stack(g, -1)
        n = (f + (g * u).sum(-1))[..., None] * u - g
        return self.radius * f, n / n.norm(dim=-1, keepdim=True)


def _radii(case, rng):
    if case["mesh"] == "sphere":
        return [_Radius(case["radius"], 0.0, rng)]
    if case["mesh"] == "star":
        return [_Radius(case["radius"], 0.08, rng)]
    return [_Radius(case["radius"] * 200.0 / 230.0, 0.01, rng), _Radius(case["radius"], 0.01, rng)]


def _panels(case, seed):
    """Panels in octree order as tensors on the GPU (vertices (N, 3, 3), normals, areas), and the surfaces' radii."""
    rng = np.random.default_rng([seed, 1])
    radii = _radii(case, rng)
    u = _unit_sphere("sphere" if case["mesh"] == "sphere" else "octa", case["size"])
    vs, ns = [], []
    for k, r in enumerate(radii):
        f, n = r(u, normal=True)
        v = f[..., None] * u
        if len(radii) == 2 and k == 0:   # the inner surface faces the cavity
            v, n = v[:, [0, 2, 1]], -n[:, [0, 2, 1]]
        vs.append(v)
        ns.append(n)
    v, n = torch.cat(vs), torch.cat(ns)
    if case["drop"]:
        keep = np.setdiff1d(np.arange(len(v)), rng.choice(len(v), case["drop"], replace=False))
        keep = torch.from_numpy(keep).cuda()
        v, n = v[keep], n[keep]
    n = n[:, 0] / 2 + (n[:, 1] + n[:, 2]) / 4
    n = n / n.norm(dim=1, keepdim=True)
    area = 0.5 * torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]).norm(dim=1)
    # octree order: digits ix + 2 iy + 4 iz of the centroid's cells, level by level
    third = 0.33333333333333333333333333
    c = third * ((v[:, 0] + v[:, 1]) + v[:, 2])
    lo, up = v.reshape(-1, 3).min(0).values, v.reshape(-1, 3).max(0).values
    side = float((up - lo).max())
    cell, key = torch.zeros_like(c), torch.zeros(len(v), dtype=torch.int64, device="cuda")
    for _ in range(case["depth"]):
        bit = c > lo + (cell + 0.5) * side
        cell = 2 * cell + bit
        key = key * 8 + (bit * torch.tensor([1, 2, 4], device="cuda")).sum(1)
        side *= 0.5
    order = torch.sort(key, stable=True).indices
    return v[order].contiguous(), n[order].contiguous(), area[order].contiguous(), radii


def _charge_set(case, radii, seed):
    rng = np.random.default_rng([seed, 2])
    m = case["charges"]
    u = rng.normal(size=(m, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    ut = torch.from_numpy(u).cuda()
    outer = radii[-1](ut).cpu().numpy() - 1.4   # at least 1.4 A inside the surface
    inner = radii[0](ut).cpu().numpy() + 1.4 if len(radii) == 2 else np.zeros(m)
    r = (inner ** 3 + (outer ** 3 - inner ** 3) * rng.random(m)) ** (1.0 / 3.0)
    q = rng.normal(0.0, 0.4, m)
    q -= (q.sum() + 5.0) / m
    return ChargeSet(pos=u * r[:, None], q=q, radius=np.full(m, 1.5))


def _params(case):
    return lib.params(order=case["order"], depth=case["depth"], sep_ratio=case["mac"], eps1=case["eps1"], eps2=EPS2,
                      kappa=KAPPA, quad_order=case["q"],
                      precision=lib.MIXED if case["precision"] == "mixed" else lib.FP64)


def _panel_set(v, n, area):
    v, n, area = (x.cpu().numpy() for x in (v, n, area))
    return PanelSet(v, n, area, np.arange(len(area), dtype=np.int32))


def _density(v, seed):
    """A density of a Krylov vector's kind: smooth over the surface with a rough part."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = v.mean(1)
    c = c / c.norm(dim=1).max()
    parts = []
    for _ in range(2):
        w = 4.0 * torch.randn(3, generator=g, device="cuda", dtype=F64)
        parts.append(torch.cos(c @ w + 1.0) + 0.3 * torch.randn(len(v), generator=g, device="cuda", dtype=F64))
    return torch.cat(parts).contiguous()


# ---------------------------------------------------------------------------------------------------------------------
# the passes
# ---------------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    v, n, area, radii = _panels(case, seed)
    panels = _panel_set(v, n, area)
    charges = _charge_set(case, radii, seed) if case["charges"] else None
    st = {"case": case, "panels": panels, "charges": charges}
    kind = case["kind"]
    if kind == "program":
        st["rhs"] = torch.empty(2 * panels.n, dtype=F64, device="cuda")
        return st
    st["surface"] = s = lib.Surface(panels, _params(case), charges, direct=case["direct"])
    if kind == "matvec":
        st["x"] = _density(v, seed)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "solve":
        s.precond_setup(case["precond"])
        st["b"] = torch.from_numpy(s.rhs(use_tree=False)).cuda()
        st["x"] = torch.empty_like(st["b"])
    elif kind == "walks":
        st["sigma"] = _density(v, seed)
        st["rhs"] = torch.empty_like(st["sigma"])
    else:
        s.precond_setup(case["precond"])
        st["q"] = torch.from_numpy(charges.q).cuda().requires_grad_()
        st["pos"] = torch.from_numpy(charges.pos).cuda().requires_grad_()
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "matvec":
        call = st["surface"].matvec_adjoint if case["adjoint"] else st["surface"].matvec
        call(st["x"].data_ptr(), y=st["y"].data_ptr(), on_device=1)
        return st["y"]
    if kind == "solve":
        st["x"].copy_(st["b"])   # the usual initial guess
        torch.cuda.current_stream().synchronize()   # the library works on its own stream
        st["surface"].solve(st["b"].data_ptr(), st["x"].data_ptr(), restart=10, maxit=100, tol=case["tol"], on_device=1)
        return st["x"]
    if kind == "walks":
        st["surface"].rhs(use_tree=True, out=st["rhs"].data_ptr(), on_device=1)
        return {"rhs": st["rhs"], "energy": KCAL * st["surface"].energy_raw(st["sigma"].data_ptr(), on_device=1)}
    if kind == "gradient":
        st["q"].grad = st["pos"].grad = None
        e = SolvationEnergy.apply(st["q"], st["pos"], st["surface"], 10, 200, case["tol"])
        e.backward()
        return {"energy": e.detach(), "q": st["q"].grad, "pos": st["pos"].grad}
    s = lib.Surface(st["panels"], _params(case), st["charges"])
    s.precond_setup(case["precond"])
    b = st["rhs"]
    s.rhs(use_tree=False, out=b.data_ptr(), on_device=1)   # the tree pays above 2e11 panel-charge pairs
    x = b.clone()
    torch.cuda.current_stream().synchronize()
    s.solve(b.data_ptr(), x.data_ptr(), restart=10, maxit=100, tol=case["tol"], on_device=1)
    e = KCAL * s.energy_raw(x.data_ptr(), on_device=1)
    s.close()
    return {"sigma": x, "energy": e}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far results may differ
# ---------------------------------------------------------------------------------------------------------------------

def _count(case):
    surfaces = 2 if case["mesh"] == "shell" else 1
    n = 20 * 4 ** case["size"] if case["mesh"] == "sphere" else 8 * surfaces * case["size"] ** 2
    return n - case["drop"], surfaces


def work(case):
    """Panel pairs from the mean leaf of a smooth closed surface (4.4 * 4^depth leaves) and the leaves that the acceptance
    ratio leaves near (15 / ratio^2); 45 operations for a pair in one direction, half of what both directions need
    together; 8 binom(p + 6, 6) for each interacting cube, about 60 of a leaf at ratio 0.8; 12 for a panel and a charge."""
    n, surfaces = _count(case)
    m, q = case["charges"], case["q"]
    leaves = min(4.4 * 4 ** case["depth"] * (1.0 if surfaces == 1 else 1.76), n)
    near = n * min(15.0 / case["mac"] ** 2 * n / leaves, n) * q ** 4
    m2l = min(leaves * 60 * (0.8 / case["mac"]) ** 4, leaves * leaves) * 8 * math.comb(case["order"] + 6, 6)
    product = 45.0 * n * n if case["direct"] else 45.0 * near + m2l
    geometry, vectors = 8 * 13 * n, 8 * 2 * n
    walk = n * min(m, 300) * 12.0
    kind = case["kind"]
    if kind == "matvec":
        return {"bytes": geometry + 2 * vectors, "flops": product}
    if kind == "walks":
        return {"bytes": geometry + 2 * vectors + 32 * m, "flops": 2 * walk}
    # block LU: blocks of about four leaves, two unknowns a panel; around ten products a solve
    rows = min(8.0 * n / leaves, 2.0 * n)
    inverse = 2.0 * n * rows
    steps = 10
    solve = {"bytes": geometry + steps * inverse * 4 + 3 * vectors, "flops": steps * (product + 2 * inverse)}
    if kind == "solve":
        return solve
    if kind == "gradient":
        return {"bytes": 2 * solve["bytes"] + 64 * m, "flops": 2 * solve["flops"] + 3 * 20.0 * n * m}
    return {"bytes": solve["bytes"] + 32 * m, "flops": solve["flops"] + walk + 15.0 * n * m + 2.0 * inverse * rows}


def tolerance(case):
    # measured with the sums of panel pairs and of interacting cubes in another order: up to 4e-6 in 32 bits, 1e-15 in
    # 64; the walks in 32 bits are 3e-7 from those in 64
    mixed = case["precision"] == "mixed"
    if case["kind"] == "matvec":
        return {"rel": 1e-5 if mixed else 1e-12}
    if case["kind"] == "walks":
        return {"rel": 2e-6 if mixed else 1e-12}
    # iterated until the residual is below tol: the last step may fall on either side of it
    return {"rel": 10 * case["tol"], "max": 1000 * case["tol"]}


# ---------------------------------------------------------------------------------------------------------------------
# the same values in 64 bits: every panel pair and every charge summed directly
# ---------------------------------------------------------------------------------------------------------------------

def _kernels(r, nx, ny, eps):
    """The four kernels at r = x - y: G0 - Gk, eps dGk/dny - dG0/dny, dGk/dnx / eps - dG0/dnx, d2(Gk - G0)/dnx dny."""
    r2 = (r * r).sum(-1)
    d = torch.sqrt(r2)
    g0 = 1.0 / (4.0 * math.pi * d)
    e = torch.exp(-KAPPA * d)
    c = (KAPPA * d + 1.0) * e
    ix, iy, ip = (nx * r).sum(-1), (ny * r).sum(-1), (nx * ny).sum(-1)
    dy, dx = iy * g0 / r2, ix * g0 / r2
    dd = (ip * g0 - 3.0 * dy * ix) / r2
    return torch.stack([g0 * (1.0 - e), (eps * c - 1.0) * dy, (c / eps - 1.0) * dx,
                        (c - 1.0) * dd - KAPPA * KAPPA * e * ix * dy])


def _gauss(q):
    t, w = np.polynomial.legendre.leggauss(q)
    return ((t + 1.0) / 2.0).tolist(), (w / 2.0).tolist()


def _touching(v):
    """Panel pairs (X, Y) that share a vertex, X itself among them, and the corners' numbers (N, 3)."""
    n = len(v)
    ids = torch.unique(v.reshape(-1, 3) + 0.0, dim=0, return_inverse=True)[1]
    by = torch.argsort(ids, stable=True)
    count = torch.bincount(ids)
    first = torch.cumsum(count, 0) - count
    pairs = [torch.arange(n, device=v.device) * (n + 1)]
    owner = torch.arange(3 * n, device=v.device) // 3
    for k in range(int(count.max())):
        ok = k < count[ids]
        other = by[(first[ids] + k).clamp(max=3 * n - 1)] // 3
        pairs.append((owner * n + other)[ok])
    p = torch.unique(torch.cat(pairs))
    return p // n, p % n, ids.reshape(n, 3)


def _touching_values(x, y, ids, v, normal, area, q, eps):
    """Sauter's and Schwab's rules for panels with a common vertex, a common edge, and for a panel with itself."""
    t, w = _gauss(q)
    out = torch.zeros(4, len(x), dtype=F64, device=v.device)
    same = ids[x][:, :, None] == ids[y][:, None, :]
    n1 = same.any(2).int().argmax(1)
    n2 = same[torch.arange(len(x), device=v.device), n1].int().argmax(1)
    step = torch.arange(3, device=v.device)
    ix, iy = (n1[:, None] + step) % 3, (n2[:, None] + step) % 3
    row = torch.arange(len(x), device=v.device)[:, None]
    vx, vy = v[x][row, ix], v[y][row, iy]     # corners from the common one on
    jx, jy = ids[x][row, ix], ids[y][row, iy]
    fwd, back = jx[:, 1] == jy[:, 2], jx[:, 2] == jy[:, 1]
    self_ = x == y

    def add(sel, offsets, weight):
        nx, ny = normal[x[sel]], normal[y[sel]]
        for r in offsets:
            out[:, sel] += weight * _kernels(r, nx, ny, eps)

    sel = self_.nonzero()[:, 0]
    a, b = v[x[sel], 1] - v[x[sel], 0], v[x[sel], 2] - v[x[sel], 1]
    for i in range(q):
        for j in range(q):
            o = t[i] * (1.0 - t[j])
            for k in range(q):
                e, f = t[k], 1.0 - t[k]
                r = [e * a + b, f * b - e * a, a + e * b]
                add(sel, [o * s * d for d in r for s in (1.0, -1.0)], o * t[i] ** 2 * t[j] * w[i] * w[j] * w[k])
    # (w of the innermost variable that the integrand does not depend on adds up to one)
    sel = (~self_ & ~fwd & ~back).nonzero()[:, 0]
    a, a0 = vx[sel, 1] - vx[sel, 0], vx[sel, 2] - vx[sel, 1]
    b, b0 = vy[sel, 1] - vy[sel, 0], vy[sel, 2] - vy[sel, 1]
    for i in range(q):
        for j in range(q):
            for k in range(q):
                for m in range(q):
                    o, e1, e2, e3 = t[i], t[j], t[k], t[m]
                    add(sel, [o * (a + e2 * a0 - e1 * (b + e3 * b0)), o * (e1 * (a + e3 * a0) - (b + e2 * b0))],
                        o ** 3 * e1 * w[i] * w[j] * w[k] * w[m])
    for which, sel in ((0, (~self_ & back).nonzero()[:, 0]), (1, (~self_ & fwd & ~back).nonzero()[:, 0])):
        if which:    # the common edge is X's first and Y's last from the common corner on
            a, b, c = vx[sel, 1] - vx[sel, 0], vx[sel, 2] - vx[sel, 1], vy[sel, 2] - vy[sel, 1]
        else:        # X's last and Y's first
            a, b, c = vx[sel, 0] - vx[sel, 2], vy[sel, 1] - vy[sel, 2], vx[sel, 1] - vx[sel, 2]
        for i in range(q):
            for j in range(q):
                o = t[i] * t[j]
                for k in range(q):
                    for m in range(q):
                        e1, e2 = t[k], t[m]
                        e3, f1, f2 = e1 * e2, 1.0 - e1, 1.0 - e2
                        f3 = 1.0 - e3
                        add(sel, [o * (e1 * (a + e2 * b) + f1 * c), o * (e1 * (b + e2 * a) + f3 * c),
                                  o * (f1 * a + b + e3 * c), o * (e1 * (e2 * b - f2 * a) + c),
                                  o * (e3 * b - f3 * a + e1 * c), o * (e1 * b - f1 * a + e3 * c)],
                            o * o * t[j] * e1 * w[i] * w[j] * w[k] * w[m])
    return out * (4.0 * area[x] * area[y])


def _points(v, q):
    """Quadrature points of every panel and their weights (without twice the panel's area)."""
    t, w = _gauss(q)
    for i in range(q):
        for j in range(q):
            yield v[:, 0] + t[i] * ((v[:, 1] - v[:, 0]) + t[j] * (v[:, 2] - v[:, 1])), t[i] * w[i] * w[j]


def _matrix(case, v, normal, area):
    """D - K, dense."""
    n, eps, q = len(v), EPS2 / case["eps1"], case["q"]
    A = torch.empty(2 * n, 2 * n, dtype=F64, device="cuda")
    pts = list(_points(v, q))
    x, y, ids = _touching(v)
    values = _touching_values(x, y, ids, v, normal, area, q, eps)
    step = max(1, 8_000_000 // n)
    for i in range(0, n, step):
        s = slice(i, min(n, i + step))
        k = torch.zeros(4, s.stop - s.start, n, dtype=F64, device="cuda")
        for px, wx in pts:
            for py, wy in pts:
                r = px[s, None] - py[None]
                k += wx * wy * _kernels(r, normal[s, None], normal[None], eps)
        k *= 4.0 * area[s, None] * area
        mine = (x >= s.start) & (x < s.stop)
        k[:, x[mine] - s.start, y[mine]] = values[:, mine]
        A[s, :n], A[s, n:] = -k[1], -k[0]
        A[n + s.start:n + s.stop, :n], A[n + s.start:n + s.stop, n:] = -k[3], -k[2]
    A.diagonal().add_(torch.cat([(1.0 + eps) / 2.0 * area, (1.0 + 1.0 / eps) / 2.0 * area]))
    return A


def _charge_sums(case, v, normal, area, q, pos, energy):
    """The right-hand side, or the energy's weights, of charges q at pos (2N values)."""
    eps = EPS2 / case["eps1"]
    out = []
    step = max(1, 40_000_000 // len(q))
    for i in range(0, len(v), step):
        s = slice(i, i + step)
        a, b = 0.0, 0.0
        for p, w in _points(v[s], case["q"]):
            r = p[:, None] - pos[None]
            d2 = (r * r).sum(-1)
            d = torch.sqrt(d2)
            dn = -(normal[s, None] * r).sum(-1) / (d2 * d)
            if energy:
                e = torch.exp(-KAPPA * d)
                a = a + w * ((eps * (KAPPA * d + 1.0) * e - 1.0) * dn) @ q
                b = b + w * ((1.0 - e) / d) @ q
            else:
                a, b = a + w * (1.0 / d) @ q, b + w * dn @ q
        c = 2.0 * area[s] / (4.0 * math.pi)
        out.append(torch.stack([c * a, c * b]) / (1.0 if energy else case["eps1"]))
    return torch.cat(out, 1).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    n, _ = _count(case)
    if kind != "walks" and n > DENSE_MAX:
        return None
    v, normal, area, radii = _panels(case, seed)
    sums = functools.partial(_charge_sums, case, v, normal, area)
    if case["charges"]:
        ch = _charge_set(case, radii, seed)
        q, pos = torch.from_numpy(ch.q).cuda(), torch.from_numpy(ch.pos).cuda()
    if kind == "walks":
        sigma = _density(v, seed)
        return {"rhs": sums(q, pos, False), "energy": KCAL * float(sums(q, pos, True) @ sigma)}
    A = _matrix(case, v, normal, area)
    if kind == "matvec":
        x = _density(v, seed)
        return A.T @ x if case["adjoint"] else A @ x
    lu, piv = torch.linalg.lu_factor(A)
    del A
    sigma = torch.linalg.lu_solve(lu, piv, sums(q, pos, False)[:, None])
    if kind == "solve":
        return sigma[:, 0]
    e = sums(q, pos, True)
    if kind == "program":
        return {"sigma": sigma[:, 0], "energy": KCAL * float(e @ sigma[:, 0])}
    lam = torch.linalg.lu_solve(lu, piv, e[:, None], adjoint=True)[:, 0]
    q.requires_grad_()
    pos.requires_grad_()
    (KCAL * (sums(q, pos, True) @ sigma[:, 0] + sums(q, pos, False) @ lam)).backward()
    return {"energy": KCAL * float(e @ sigma[:, 0]), "q": q.grad, "pos": pos.grad}
