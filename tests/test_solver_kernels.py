"""Preconditioner, GMRES, translation and charge-tree kernels at the sizes where their dispatch changes, against the FP64
restatement oracle.

Tolerances: FP64 operators 1e-12 and block inverses 1e-11 relative L2, as for the golden cases; block inverses of mixed
contexts 1e-4 (FP32 inverses of well-conditioned blocks: rows * 2^-24 <= 1536 * 6e-8); mixed operators 5e-6.
"""
import concurrent.futures
import functools

import numpy as np
import pytest
import scipy.linalg

from conftest import rel_l2
from fabipb_b200 import lib, meshgen, meshio
from oracle import oracle as O
from test_near_kernels import cut_sphere

pytestmark = pytest.mark.gpu


def patch_and_far_panel(panels):
    """`panels` faces around a pole of the 5,120-panel sphere and one face far away: at depth 1 the patch is one leaf."""
    unit, faces = meshgen.icosphere(4)
    pan = meshio.build_panels(20.0 * unit, unit, faces)
    z = pan.vtx[:, :, 2].mean(1)
    keep = np.sort(np.argsort(-z)[:panels])
    far = int(np.argmin(z))
    vtx = np.concatenate([pan.vtx[keep], pan.vtx[far:far + 1] + np.array([300.0, 300.0, -300.0])])
    keep = np.r_[keep, far]
    return meshio.PanelSet(vtx, pan.normal[keep], pan.area[keep], pan.face_index[keep])


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-11), (lib.MIXED, 1e-4)])
@pytest.mark.parametrize("panels", [1, 3, 4, 8, 9, 17, 191, 192, 193, 384, 385, 768, 769])
def test_block_inverse_classes(panels, precision, tol):
    """Blocks of 2 * panels + 2 rows (the patch and the far panel) on both sides of every class of the inversion, and of
    every batch of the application.  Their pivots all lie on the diagonal; test_block_inverse_pivoting has others."""
    pan = patch_and_far_panel(panels)
    opts = dict(order=2, depth=1, height=1)
    s, o = lib.Surface(pan, lib.params(precision=precision, **opts)), O.Oracle(pan, O.make_params(**opts))
    assert sorted(s.leaf_layout()[1]) == [1, panels]
    s.precond_setup(2)
    o.precond_setup(2)
    b = np.random.default_rng(panels).standard_normal(2 * s.n)
    assert rel_l2(s.precond_apply(b), o.precond_apply(b)) < tol


def three_sheets(panels):
    """Three parallel sheets of a third of the panels each, 0.3 and 0.2 panel widths apart: the double-layer values of
    facing panels are above the diagonal, and partial pivoting takes a panel's column to another sheet's row."""
    unit, faces = meshgen.icosphere(4)
    pan = meshio.build_panels(20.0 * unit, unit, faces)
    order, width = np.argsort(-pan.vtx[:, :, 2].mean(1)), np.sqrt(pan.area.mean())
    parts = []
    for k, r in enumerate(1.0 + width / 20.0 * np.array([0.0, 0.3, 0.5])):
        a = np.sort(order[:(panels + 2 - k) // 3])
        parts.append((r * pan.vtx[a], pan.normal[a], r * r * pan.area[a]))
    return meshio.PanelSet(*(np.concatenate(x) for x in zip(*parts)), np.arange(panels, dtype=np.int32))


@functools.lru_cache(maxsize=None)
def moved_pivots(panels):
    """Columns of the three sheets' block whose pivot's own column has yet another pivot, by LAPACK on the host."""
    o = O.Oracle(three_sheets(panels), O.make_params(order=2, depth=1, height=1))
    n, area, eps = o.n, o.area(), 80.0
    K = np.array([[o.panel_ia0(x, y) for y in range(n)] for x in range(n)])
    A = -np.block([[K[..., 1], K[..., 3]], [K[..., 0], K[..., 2]]])
    A[np.diag_indices(2 * n)] += np.r_[(1 + eps) / 2 * area, (1 + 1 / eps) / 2 * area]
    b = np.random.default_rng(0).standard_normal(2 * n)
    o.precond_setup(2)
    assert rel_l2(np.linalg.solve(A, b), o.precond_apply(b)) < 1e-12   # the block that the preconditioner inverts
    perm = np.arange(2 * n)
    for k, j in enumerate(scipy.linalg.lu_factor(A)[1]):
        perm[[k, j]] = perm[[j, k]]
    return int((perm[perm] != np.arange(2 * n)).sum())


@pytest.mark.parametrize("panels", [17, 192, 193, 384, 385, 768, 769])
@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-11), (lib.MIXED, 2e-3)])
def test_block_inverse_pivoting(panels, precision, tol):
    """Blocks of 2 * panels rows, the last and first of every class, whose pivots lie off the diagonal, in cycles of
    three and more.  The application against the oracle: the blocks' condition is 550, so an FP32 inverse is within
    550 * 2^-24 * sqrt(1538) = 1.3e-3.  The transposed application by the steps of the adjoint solve of the direct
    operator, of which the block is all: as many as the forward solve takes, 5 or 6; with the index lists left out or
    exchanged it takes 15 to 26."""
    assert moved_pivots(panels) > 1.5 * panels
    pan = three_sheets(panels)
    opts = dict(order=2, depth=1, height=1)
    s, o = lib.Surface(pan, lib.params(precision=precision, **opts), direct=True), O.Oracle(pan, O.make_params(**opts))
    s.precond_setup(2)
    o.precond_setup(2)
    b = np.random.default_rng(panels).standard_normal(2 * s.n)
    assert rel_l2(s.precond_apply(b), o.precond_apply(b)) < tol
    rng = np.random.default_rng(1)
    s.set_charges(meshio.ChargeSet(rng.uniform(-5, 5, (7, 3)), rng.standard_normal(7), np.ones(7)))
    _, it, _, info = s.forward(restart=30, maxit=30, tol=1e-10)
    _, _, it_t, _, info_t = s.backward(1.0, restart=30, maxit=30, tol=1e-10)
    assert info == 0 and info_t == 0 and it <= 8 and abs(it - it_t) <= 1


def patches(sizes):
    """Patches of these many panels, each in an octant of its own."""
    unit, faces = meshgen.icosphere(4)
    pan = meshio.build_panels(20.0 * unit, unit, faces)
    order = np.argsort(-pan.vtx[:, :, 2].mean(1))
    keep = [np.sort(order[:n]) for n in sizes]
    at = [300.0 * np.array([1 - 2 * (k & 1), 1 - (k & 2), 1 - (k & 4) / 2]) for k in range(len(sizes))]
    return meshio.PanelSet(np.concatenate([pan.vtx[k] + a for k, a in zip(keep, at)]),
                           *(np.concatenate([x[k] for k in keep]) for x in (pan.normal, pan.area)),
                           np.arange(sum(sizes), dtype=np.int32))


@pytest.mark.parametrize("sizes", [(12, 250), (12, 250, 500), (3, 10, 250, 260, 500, 800), (5, 300, 1601)])
def test_block_inverse_classes_together(sizes):
    """Blocks of several classes in one surface, which are inverted side by side, up to those of the library LU: FP64
    against the oracle (to 800 panels), mixed against FP64."""
    pan = patches(sizes)
    opts = dict(order=2, depth=2, height=2)
    s, m = (lib.Surface(pan, lib.params(precision=p, **opts)) for p in (lib.FP64, lib.MIXED))
    b = np.random.default_rng(len(sizes)).standard_normal(2 * s.n)
    x = []
    for t in (s, m, s):   # the third: again on a context that has a preconditioner
        t.precond_setup(2)
        x.append(t.precond_apply(b))
    assert rel_l2(x[1], x[0]) < 1e-4 and (x[2] == x[0]).all()
    if max(sizes) <= 800:
        o = O.Oracle(pan, O.make_params(**opts))
        o.precond_setup(2)
        assert rel_l2(x[0], o.precond_apply(b)) < 1e-11


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
@pytest.mark.parametrize("panels", [1, 17, 193, 385, 800])
@pytest.mark.parametrize("where", [0, -1])
def test_block_inverse_of_a_non_finite_panel(panels, where, precision):
    """A panel whose normal is 0/0 makes a row and a column of its block NaN: an error in every class, and the
    context is as good as before."""
    pan = patch_and_far_panel(panels)
    normal = pan.normal.copy()
    normal[0 if where == 0 else panels - 1] = np.nan
    s = lib.Surface(meshio.PanelSet(pan.vtx, normal, pan.area, pan.face_index),
                    lib.params(order=2, depth=1, height=1, precision=precision))
    with pytest.raises(RuntimeError, match="non-finite pivot"):
        s.precond_setup(2)
    with pytest.raises(RuntimeError, match="not set up"):
        s.precond_apply(np.ones(2 * s.n))
    s.precond_setup(3)   # the diagonal, which reads areas only
    assert np.isfinite(s.precond_apply(np.ones(2 * s.n))).all()


@pytest.mark.parametrize("panels,depth", [(5, 2), (331, 2), (643, 1)])
def test_adjoint_block_application(panels, depth):
    """The energy is quadratic in the charges, so q . dE/dq = 2 E; the transposed solve takes the forward one's steps."""
    pan = cut_sphere(panels, seed=panels)
    rng = np.random.default_rng(panels)
    ch = meshio.ChargeSet(rng.uniform(-5, 5, (7, 3)), rng.standard_normal(7), np.ones(7))
    s = lib.Surface(pan, lib.params(order=3, depth=depth, height=min(depth, 2), precision=lib.FP64), charges=ch)
    s.precond_setup(2)
    e, it, _, info = s.forward(restart=20, maxit=200, tol=1e-12)
    dq, _, it_t, _, info_t = s.backward(1.0, restart=20, maxit=200, tol=1e-12)
    assert info == 0 and info_t == 0 and abs(it - it_t) <= max(2, it // 4)
    assert abs(dq @ ch.q - 2 * e) <= 1e-9 * abs(2 * e)


def graded_spheres():
    """Five 80-panel spheres whose panel areas span 1 to 0.1: without a preconditioner a hundred steps and more."""
    unit, faces = meshgen.icosphere(1)
    parts = []
    for i in range(5):
        at = np.array([60 * np.cos(0.7 * i), 60 * np.sin(0.7 * i), 10 * i]) * 0.75 ** i
        parts.append(meshio.build_panels(20 * 0.75 ** i * unit + at, unit, faces))
    return meshio.PanelSet(*(np.concatenate([getattr(p, f) for p in parts])
                             for f in ("vtx", "normal", "area", "face_index")))


@pytest.mark.parametrize("restart", [1, 2, 10, 63, 64, 65, 90])
def test_gmres_restart_lengths(restart):
    """A hundred steps in cycles of one column, of a few and of more than one staged group of columns, ended before they
    converge: the oracle's iterate.  A relative change of 1e-16 in the right-hand side moves it by 1e-10 at restart 1 and
    by 1e-12 above; operators that agree to 1e-15 leave it within 1e-8."""
    pan = graded_spheres()
    opts = dict(order=3, depth=3, height=2)
    s, o = lib.Surface(pan, lib.params(precision=lib.FP64, **opts)), O.Oracle(pan, O.make_params(**opts))
    b = np.random.default_rng(3).standard_normal(2 * s.n)
    s.precond_setup(-1)
    o.precond_setup(-1)
    x, it, res, info = s.solve(b, b.copy(), restart=restart, maxit=100, tol=1e-14)
    xr, itr, resr, infor = o.gmres(b, b.copy(), restart, 100, 1e-14)
    assert (it, info) == (itr, infor) and abs(res - resr) <= 1e-6 * resr
    assert rel_l2(x, xr) < 1e-8


def cloud():
    """49 ellipsoids of 32 panels whose areas spread evenly over 1 to 65: without a preconditioner a decade in 65 steps."""
    unit, faces = meshgen.octasphere(2)
    rng = np.random.default_rng(1)
    parts = []
    for i in range(49):
        r, axes = 4 * np.exp(rng.uniform(np.log(0.2), 0)), np.exp(rng.uniform(-0.4, 0.4, 3))
        normal = unit / axes
        normal /= np.linalg.norm(normal, axis=1)[:, None]
        at = 12.0 * np.array([i % 4, i // 4 % 4, i // 16])
        parts.append(meshio.build_panels(r * unit * axes + at, normal, faces))
    return meshio.PanelSet(*(np.concatenate([getattr(p, f) for p in parts])
                             for f in ("vtx", "normal", "area", "face_index")))


def test_gmres_cycle_of_thousands_of_columns():
    """One cycle of more columns than a block's shared memory holds coefficients: every step is taken, and the iterate
    solves the system as far as 64 bits go (condition 80 * 65, so a residual below 5200 * 2^-53 * sqrt(3000) = 3e-11)."""
    s = lib.Surface(cloud(), lib.params(precision=lib.FP64, order=3, depth=3))
    s.precond_setup(-1)
    b = np.random.default_rng(4).standard_normal(2 * s.n)
    x, it, _, info = s.solve(b, np.zeros(2 * s.n), restart=3000, maxit=3000, tol=1e-300)
    assert (it, info) == (3000, 1)
    assert np.linalg.norm(b - s.matvec(x)) <= 3e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-12), (lib.MIXED, 5e-6)])
@pytest.mark.parametrize("order", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("depth", [3, 4])
def test_far_field_cube_counts(depth, order, precision, tol):
    """Fewer and more destination cubes than the M2L kernels' dispatch line."""
    unit, faces = meshgen.icosphere(4)
    pan = meshio.build_panels(20.0 * unit, unit, faces)
    opts = dict(order=order, depth=depth, height=2)
    s, o = lib.Surface(pan, lib.params(precision=precision, **opts)), O.Oracle(pan, O.make_params(**opts))
    v = np.random.default_rng(order).standard_normal(2 * s.n)
    assert rel_l2(s.apply(v, part=lib.FAR), o.far_apply(v)) < tol


@pytest.mark.parametrize("order", [1, 3, 6])
@pytest.mark.parametrize("charges", [1, 2, 33, 257, 3000])
def test_charge_tree_moments(charges, order):
    """Right-hand side by the charge tree, whose moments are formed on the device, against the oracle's tree."""
    pan = cut_sphere(300)
    rng = np.random.default_rng(charges)
    ch = meshio.ChargeSet(rng.uniform(-9, 9, (charges, 3)), rng.standard_normal(charges), np.ones(charges))
    opts = dict(order=order, depth=3, height=2)
    s = lib.Surface(pan, lib.params(precision=lib.FP64, **opts), charges=ch)
    o = O.Oracle(pan, O.make_params(**opts), charges=ch)
    assert rel_l2(s.rhs(use_tree=True), o.rhs_tree()) < 1e-12


def test_contexts_on_threads():
    """Contexts of other block sizes and orders at work on two threads: each launch asks for its own shared memory."""
    def work(case):
        sizes, order = case
        pan = patches(sizes)
        s = lib.Surface(pan, lib.params(order=order, depth=4, height=2, precision=lib.FP64))
        b = np.random.default_rng(order).standard_normal(2 * s.n)
        out = []
        for _ in range(30):
            s.precond_setup(2)
            out.append(np.r_[s.precond_apply(b), s.matvec(b)])
        return out

    cases = [((90, 250, 500), 7), ((60, 200, 400), 8)]
    with concurrent.futures.ThreadPoolExecutor(2) as pool:
        both = list(pool.map(work, cases))
    for case, out in zip(cases, both):
        alone = work(case)[0]
        assert all((x == alone).all() for x in out)
