"""The tangent fluxes take one launch at every size (on 505,120 faces too), and
<lambda, J v> = <J^T lambda, v> holds with velocity inlets and pressure outlets
(the bar of the transpose tests, 1e-12 of the sum of magnitudes)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _geometry(kind):
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import box_mesh, riemann_case
    from meshcfd_gb300.model import Case

    if kind != "duct":
        case = riemann_case(kind)[0]
    else:
        case = Case(name="duct", mesh=box_mesh(13, 7, 2.0, 1.0, split="half", jitter=0.1, seed=1))
        for c in case.boundary_conditions:
            if c.patch_name == "left":
                c.kind, c.values = "Velocity Inlet", {"density": 1.0, "temperature": 1.0 / 287.05, "velocity_x": 0.3}
            elif c.patch_name == "right":
                c.kind, c.values = "Pressure Outlet", {"pressure": 0.9}
            else:
                c.kind, c.mechanical_condition = "Wall", "Slip"
    return case.numerics, build_geometry(case.mesh, case)


@pytest.mark.parametrize("recon,launches", (("MUSCL linear", 4), ("First order", 3)))
@pytest.mark.parametrize("kind", (9, 410, "duct"))
def test_one_launch_and_transposes(cuda_device, kind, recon, launches):
    from meshcfd_gb300.adjoint import ResidualFunction
    from meshcfd_gb300.device import DeviceGeometry, make_config, primitive_to_conservative
    from meshcfd_gb300.meshes import smooth_primitive

    s, g = _geometry(kind)
    s.flux, s.limiter, s.reconstruction = "HLLC", "Van Leer", recon
    dg, cfg, n = DeviceGeometry(g), make_config(s), len(g.areas)
    U = torch.as_tensor(primitive_to_conservative(smooth_primitive(n, seed=4, amplitude=0.3), s.gamma),
                        device=cuda_device)
    rng = np.random.default_rng(5)
    lam, v = (torch.as_tensor(rng.standard_normal((n, 4)), device=cuda_device) for _ in range(2))
    jv = torch.empty_like(v)
    for _ in range(2):  # the first call allocates
        before = dg.lib.mcfd_launch_count()
        assert dg.lib.mcfd_jvp(dg.handle, C.byref(cfg), U.data_ptr(), v.data_ptr(), jv.data_ptr(),
                               torch.cuda.current_stream().cuda_stream) == 0
    assert dg.lib.mcfd_launch_count() - before == launches
    Ug = U.clone().requires_grad_(True)
    ResidualFunction.apply(Ug, dg, cfg).backward(lam)
    dg.check_status()
    a, b = float((lam * jv).sum()), float((Ug.grad * v).sum())
    assert abs(a - b) <= 1e-12 * float((lam * jv).abs().sum())
