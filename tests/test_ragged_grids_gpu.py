"""Records and gradients of the four-cells-per-thread kernels on grids that end
inside a thread's group, a block or a tile, against the float64 oracle.

Tolerance: a cell's update sums at most ``terms`` rounded products, so a step
adds at most terms * 2**-24 of the field's size and nt steps nt times that; a
gradient multiplies two such fields, which doubles it."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests._util import rel

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
NT = 80


def _models(names, shape, rng):
    z = np.arange(shape[0]).reshape((-1,) + (1,) * (len(shape) - 1))
    vp = 2000.0 + 12.0 * z + 40.0 * rng.standard_normal(shape)
    eps = 0.1 + 0.004 * z + 0.01 * rng.standard_normal(shape)
    m = dict(vp=vp, vs=vp / 1.8, rho=310.0 * vp ** 0.25, eps=eps, dlt=0.4 * eps)
    return [m[n].astype(np.float32) for n in names]


def _geometry(shape, B, rng):
    """Shots in the core (one shared cell), receivers over the whole grid, its
    corners among them."""
    ext = np.array(shape[::-1])                     # x[, y], z
    src = rng.integers(ext // 3, 2 * ext // 3, (B, len(shape)))
    src[-1] = src[0]
    rec = rng.integers(0, ext, (B, 21, len(shape)))
    rec[:, 0], rec[:, 1] = 0, ext - 1
    return src.astype(np.int64), rec.astype(np.int64)


def _check(eq, oracle, names, shape, B, order, free=False, vacuum=False, fluid=False):
    from sweep_b200 import PropTorch
    rng = np.random.default_rng(sum(shape) + 7 * order + B)
    ms = _models(names, shape, rng)
    if vacuum:                                      # a few cells without stiffness
        ms[0].reshape(-1)[rng.integers(0, ms[0].size, 5)] = 0.0
    if fluid:                                       # water above solid
        ms[1][:shape[0] // 3] = 0.0
    src, rec = _geometry(shape, B, rng)
    dh, dt, abcn = 6.0, 0.0006, 5
    t = np.arange(NT) * dt
    a = (np.pi * 30 * (t - 0.02)) ** 2
    w = ((1 - 2 * a) * np.exp(-a)).astype(np.float32)
    kw = dict(free_surface=True) if free else {}
    run = oracle(*ms, w, src, rec, dh, dt, abcn, order=order, prec="f64", **kw)
    exact = run.forward(keep_tape=True)
    residual = (rng.standard_normal(exact.shape) * np.abs(exact).max()).astype(np.float32)
    want = run.backward(residual)
    want = want[:len(ms)]                           # less the wavelet's
    s = PropTorch(eq(spatial_order=order, device=DEV), shape=shape, dh=dh, dt=dt, abcn=abcn, device=DEV, **kw)
    ts = [torch.tensor(m, device=DEV, requires_grad=True) for m in ms]
    pred = s(torch.tensor(w, device=DEV), src, rec, models=ts)
    pred.backward(torch.tensor(residual, device=DEV))
    terms = len(shape) * (2 * order + 8)
    tol = NT * terms * 2.0 ** -24
    errs = [rel(x.grad.cpu().numpy(), g.reshape(shape)) for x, g in zip(ts, want)]
    r = rel(pred.detach().cpu().numpy(), exact)
    print(f"{eq.__name__} {shape} x {B} order {order}: record {r:.1e}, gradients "
          + " / ".join(f"{e:.1e}" for e in errs) + f" (tolerance {tol:.1e}, {2 * tol:.1e})")
    assert r < tol
    assert max(errs) < 2 * tol


@pytest.mark.parametrize("shape,B,order", [
    ((11, 13), 1, 2), ((33, 32), 3, 4), ((41, 58), 6, 8), ((40, 63), 2, 14), ((65, 129), 5, 6)])
def test_vti2d(shape, B, order):
    from sweep_b200 import AcousticVTI1st
    _check(AcousticVTI1st, O.VTI2D, ("vp", "eps", "dlt", "rho"), shape, B, order)


@pytest.mark.parametrize("shape,B,order", [
    ((12, 11, 13), 1, 2), ((17, 15, 34), 5, 4), ((20, 25, 31), 2, 10)])
def test_vti3d(shape, B, order):
    from sweep_b200 import AcousticVTI1st3D
    _check(AcousticVTI1st3D, O.VTI3D, ("vp", "eps", "dlt", "rho"), shape, B, order)


@pytest.mark.parametrize("shape,order", [((33, 32), 4), ((17, 15, 34), 4)])
def test_vti_vacuum_cells(shape, order):
    """Cells with vp = 0 (and rho > 0) take no part in the misfit by vp."""
    from sweep_b200 import AcousticVTI1st, AcousticVTI1st3D
    eq, oracle = (AcousticVTI1st, O.VTI2D) if len(shape) == 2 else (AcousticVTI1st3D, O.VTI3D)
    _check(eq, oracle, ("vp", "eps", "dlt", "rho"), shape, 2, order, vacuum=True)


@pytest.mark.parametrize("shape,B,order", [
    ((11, 13), 1, 2), ((33, 32), 3, 4), ((41, 58), 6, 6), ((40, 63), 2, 14), ((65, 129), 5, 4)])
def test_acoustic2d_other_orders(shape, B, order):
    from sweep_b200 import Acoustic
    _check(Acoustic, O.Acoustic2D, ("vp",), shape, B, order)


@pytest.mark.parametrize("shape,B,order", [
    ((12, 11, 13), 1, 2), ((17, 15, 34), 5, 4), ((20, 25, 31), 2, 12)])
def test_acoustic3d_other_orders(shape, B, order):
    from sweep_b200 import Acoustic3D
    _check(Acoustic3D, O.Acoustic3D, ("vp",), shape, B, order)


@pytest.mark.parametrize("shape,B,order", [
    ((12, 11, 13), 1, 2), ((17, 15, 34), 5, 4), ((20, 25, 31), 2, 8)])
def test_elastic3d(shape, B, order):
    from sweep_b200 import Elastic3D
    _check(Elastic3D, O.Elastic3D, ("vp", "vs", "rho"), shape, B, order)


@pytest.mark.parametrize("shape,B,order,free", [
    ((11, 13), 1, 2, False), ((33, 32), 3, 4, True), ((41, 58), 6, 6, False), ((40, 63), 2, 14, False),
    ((65, 129), 5, 4, True)])
def test_elastic2d_other_orders(shape, B, order, free):
    from sweep_b200 import Elastic
    _check(Elastic, O.Elastic2D, ("vp", "vs", "rho"), shape, B, order, free)


@pytest.mark.parametrize("shape,B", [
    ((11, 13), 1), ((33, 32), 3), ((64, 129), 5), ((65, 65), 493), ((65, 65), 494)])
def test_acoustic2d_small_and_tiled(shape, B):
    """The last two sit on both sides of the 2960 tiles of 64 x 32 cells at
    which order 8 leaves its small-grid kernels (6 tiles per shot)."""
    from sweep_b200 import Acoustic
    _check(Acoustic, O.Acoustic2D, ("vp",), shape, B, 8)


@pytest.mark.parametrize("shape,B,free", [
    ((11, 13), 1, False), ((33, 32), 3, True), ((41, 58), 6, False), ((64, 129), 5, True), ((130, 350), 21, False)])
def test_elastic2d_order8(shape, B, free):
    """The last one sums the images of several shots per thread."""
    from sweep_b200 import Elastic
    _check(Elastic, O.Elastic2D, ("vp", "vs", "rho"), shape, B, 8, free)


@pytest.mark.parametrize("shape,order,free", [((33, 45), 4, False), ((33, 45), 8, True), ((17, 15, 34), 4, False)])
def test_elastic_water_layer(shape, order, free):
    """Cells with vs = 0, whose adjoint shear stress reaches no result."""
    from sweep_b200 import Elastic, Elastic3D
    eq, oracle = (Elastic, O.Elastic2D) if len(shape) == 2 else (Elastic3D, O.Elastic3D)
    _check(eq, oracle, ("vp", "vs", "rho"), shape, 2, order, free, fluid=True)
