"""The per-variable derivative kernels and the one-launch tangent fluxes at
their edges: <lambda, J v> = <J^T lambda, v> (the two are written apart, the
bar of the transpose tests, 1e-12 of the sum of magnitudes) on cells of five
and six faces, meshes of a few cells, mixed and triangular meshes with walls
and far field, and on either side of the 500,000 faces above which the
tangent fluxes launch per segment."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITERS = ("Barth-Jespersen", "Minmod", "Van Leer", "Venkatakrishnan")


def _case(kind):
    from meshcfd_gb300.meshes import periodic_case, riemann_case
    from test_gpu_polygons import _polygon_case

    if kind == "polygons":
        return _polygon_case()
    if kind[0] == "riemann":
        return riemann_case(kind[1])[0]
    return periodic_case(kind[1], kind[2], split=kind[0], jitter=0.2, seed=6)


def _check(cuda_device, kind, flux, limiter, recon="MUSCL linear"):
    import torch
    from meshcfd_gb300.adjoint import ResidualFunction
    from meshcfd_gb300.device import DeviceGeometry, make_config, primitive_to_conservative
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import smooth_primitive

    case = _case(kind)
    s = case.numerics
    s.flux, s.reconstruction, s.limiter = flux, recon, limiter
    g = build_geometry(case.mesh, case)
    dg = DeviceGeometry(g)
    cfg = make_config(s)
    n = len(g.areas)
    U = torch.as_tensor(primitive_to_conservative(smooth_primitive(n, seed=4, amplitude=0.6), s.gamma),
                        device=cuda_device)
    rng = np.random.default_rng(5)
    lam = torch.as_tensor(rng.standard_normal((n, 4)), device=cuda_device)
    v = torch.as_tensor(rng.standard_normal((n, 4)), device=cuda_device)
    Ug = U.clone().requires_grad_(True)
    ResidualFunction.apply(Ug, dg, cfg).backward(lam)
    jv = torch.empty_like(v)
    assert dg.lib.mcfd_jvp(dg.handle, C.byref(cfg), U.data_ptr(), v.data_ptr(), jv.data_ptr(),
                           torch.cuda.current_stream().cuda_stream) == 0
    dg.check_status()
    a, b = float((lam * jv).sum()), float((Ug.grad * v).sum())
    assert abs(a - b) <= 1e-12 * float((lam * jv).abs().sum())


@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("kind", ("polygons", ("none", 3, 3), ("half", 9, 7), ("riemann", 2), ("riemann", 9)))
def test_products_are_transposes(cuda_device, kind, limiter):
    for flux in ("HLLC", "Roe", "Rusanov"):
        _check(cuda_device, kind, flux, limiter)


@pytest.mark.parametrize("flux", ("HLLC", "Roe", "Rusanov"))
def test_first_order_products_are_transposes(cuda_device, flux):
    for kind in ("polygons", ("riemann", 5)):
        _check(cuda_device, kind, flux, "Minmod", "First order")


@pytest.mark.parametrize("n", (400, 410))  # 480,800 and 505,120 faces
def test_products_are_transposes_on_large_meshes(cuda_device, n):
    _check(cuda_device, ("riemann", n), "Roe", "Barth-Jespersen")
