"""The near-field kernels at the sizes where their tiling can go wrong, against the FP64 restatement oracle.

Surfaces are cut from a 1,280-panel sphere, so that leaves hold anything from one panel to more than a tile and the
special-pair table has open edges.  Tolerances: FP64 1e-12 relative L2, the parity tolerance of the golden cases; mixed
5e-6 (FP32 pair terms).
"""
import numpy as np
import pytest

from conftest import rel_l2
from fabipb_b200 import lib, meshgen, meshio
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def cut_sphere(panels, seed=0):
    """`panels` faces of the 1,280-panel sphere: a patch, so that some leaves are full and some hold one panel."""
    unit, faces = meshgen.icosphere(3)
    pan = meshio.build_panels(20.0 * unit, unit, faces)
    axis = np.random.default_rng(seed).normal(size=3)
    keep = np.sort(np.argsort(-(pan.vtx.mean(1) @ axis))[:panels])
    return meshio.PanelSet(pan.vtx[keep], pan.normal[keep], pan.area[keep], pan.face_index[keep])


def both(pan, precision, **opts):
    s = lib.Surface(pan, lib.params(precision=precision, **opts))
    o = O.Oracle(pan, O.make_params(**opts))
    return s, o


def check(s, o, tol):
    rng = np.random.default_rng(7)
    u, v = rng.standard_normal(2 * s.n), rng.standard_normal(2 * s.n)
    k = o.near_apply(v)
    assert rel_l2(s.apply(v, part=lib.NEAR), k) < tol
    kt = s.apply_adjoint(u, part=lib.NEAR)   # the transposed operator, by duality
    assert abs(u @ k - kt @ v) <= tol * np.linalg.norm(u) * np.linalg.norm(k)


@pytest.mark.parametrize("q", [2, 3])
@pytest.mark.parametrize("panels,depth", [(2, 2), (37, 2), (319, 3), (640, 2)])
def test_quadrature_near_field(panels, depth, q):
    check(*both(cut_sphere(panels), lib.FP64, order=3, depth=depth, quad_order=q), 1e-12)


@pytest.mark.parametrize("kappa", [0.0, 1e-3, 40.0])
def test_quadrature_near_field_screening(kappa):
    """No screening, and so much that e^{-kappa r} underflows for most pairs."""
    check(*both(cut_sphere(200), lib.FP64, order=3, depth=3, quad_order=2, kappa=kappa), 1e-12)


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-12), (lib.MIXED, 5e-6)])
@pytest.mark.parametrize("panels,depth", [(2, 2), (33, 2), (319, 1), (641, 1), (1279, 2), (1280, 3)])
def test_near_field_tiles(panels, depth, precision, tol):
    """Leaves of one panel up to several tiles: groups and tiles that end anywhere, tasks on warps and half-warps, leaves
    below the tasks' least size, whole leaves split over tasks."""
    check(*both(cut_sphere(panels, seed=panels), precision, order=3, depth=depth, height=min(2, depth)), tol)


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-12), (lib.MIXED, 5e-6)])
@pytest.mark.parametrize("kappa", [0.0, 40.0])
def test_near_field_screening(kappa, precision, tol):
    check(*both(cut_sphere(900), precision, order=3, depth=2, kappa=kappa), tol)


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-12), (lib.MIXED, 5e-6)])
def test_near_field_zero_densities(precision, tol):
    """A density with one half zero, and one of a single panel."""
    s, o = both(cut_sphere(700), precision, order=3, depth=2)
    for v in (np.r_[np.zeros(s.n), np.ones(s.n)], np.r_[np.ones(s.n), np.zeros(s.n)], np.eye(2 * s.n)[3]):
        assert rel_l2(s.apply(v, part=lib.NEAR), o.near_apply(v)) < tol


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-12), (lib.MIXED, 5e-6)])
@pytest.mark.parametrize("panels,depth", [(3, 2), (127, 2), (129, 3), (641, 2), (1279, 3)])
def test_direct_operator_parts(panels, depth, precision, tol):
    """The direct context's parts (runs of 128 panels in FP64, leaves in mixed contexts) against the oracle with no far
    field: an acceptance ratio so small that every leaf pair is near."""
    pan = cut_sphere(panels, seed=panels)
    opts = dict(order=3, depth=depth, sep_ratio=1e-9)
    s = lib.Surface(pan, lib.params(precision=precision, **opts), direct=True)
    check(s, O.Oracle(pan, O.make_params(**opts)), tol)


@pytest.mark.parametrize("panels,doubled", [(641, 40), (1280, 100)])
@pytest.mark.parametrize("sym", ["1", "0"])
def test_direct_operator_coincident_panels(panels, doubled, sym, monkeypatch):
    """Doubled faces whose two panels fall into different runs of 128: their one-point term is 0 and their
    special-pair value stands alone, in the symmetric tasks and in the ordered passes."""
    monkeypatch.setenv("FABIPB_B200_NEAR_SYM", sym)
    pan = cut_sphere(panels, seed=panels)
    twice = np.r_[np.arange(panels), np.linspace(0, panels - 1, doubled).astype(int)]
    pan = meshio.PanelSet(pan.vtx[twice], pan.normal[twice], pan.area[twice], np.arange(len(twice), dtype=np.int32))
    opts = dict(order=3, depth=1, height=1, sep_ratio=1e-9)
    s = lib.Surface(pan, lib.params(precision=lib.FP64, **opts), direct=True)
    run = np.empty(len(twice), int)
    run[s.panel_order()] = np.arange(len(twice)) // 128
    assert (run[twice[panels:]] != run[panels:]).any()
    check(s, O.Oracle(pan, O.make_params(**opts)), 1e-12)


@pytest.mark.parametrize("precision,tol", [(lib.FP64, 1e-13), (lib.MIXED, 5e-6)])
def test_direct_operator_long_parts(precision, tol, monkeypatch):
    """Parts and chunks above 256 panels, where the direct context's scratch bound sets them: the symmetric tasks
    against the ordered passes of the same context.  FP64: two orders of 1e5 sums of random sign, 2^-53 * sqrt(1e5)."""
    unit, faces = meshgen.octasphere(112)
    pan = meshio.build_panels(20.0 * unit, unit, faces)
    v = np.random.default_rng(5).standard_normal(2 * pan.n)
    out = []
    for sym in ("1", "0"):
        monkeypatch.setenv("FABIPB_B200_NEAR_SYM", sym)
        s = lib.Surface(pan, lib.params(precision=precision, order=3, depth=3, height=2), direct=True)
        out.append(s.apply(v, part=lib.NEAR))
        out.append(s.apply_adjoint(v, part=lib.NEAR))
        s.close()
    assert rel_l2(out[0], out[2]) < tol and rel_l2(out[1], out[3]) < tol
