"""Tuned flux shapes on meshes whose fluxes take one launch by default: a block
size is taken by that launch, several faces a thread by a launch per face
segment (counted), and every shape gives the default's bits, on every kind of
boundary segment (in fma mode, where each kernel contracts its own products,
the same to 1e-13 of the largest entry)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

R_GAS = 287.05
VELOCITY = ("Velocity Inlet", {"density": 1.0, "velocity_x": 0.3, "velocity_y": 0.0, "pressure": 1.0})
OUTLET = ("Pressure Outlet", {"pressure": 0.9})
TOTAL = ("Pressure Inlet", {"pressure": 1.2, "temperature": 1.1 / R_GAS, "velocity_x": 1.0, "velocity_y": 0.1})
FLOW_IN = ("Mass Flow Inlet", {"mass_flow": 0.3, "temperature": 1.1 / R_GAS, "velocity_x": 1.0, "velocity_y": 0.0})
FLOW_OUT = ("Mass Flow Outlet", {"mass_flow": 0.3})
# kind: segments with faces (interior among them)
SEGMENTS = {"velocity": 4, "total": 4, "flow": 3, "riemann": 3, "vortex": 2}


def _geometry(kind):
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import box_mesh, riemann_case, smooth_primitive, vortex_case
    from meshcfd_gb300.model import Case

    if kind == "riemann":
        case = riemann_case(48)[0]
    elif kind == "vortex":
        case = vortex_case(50, split="half")[0]
    else:
        left, right = {"velocity": (VELOCITY, OUTLET), "total": (TOTAL, OUTLET), "flow": (FLOW_IN, FLOW_OUT)}[kind]
        case = Case(name="duct", mesh=box_mesh(60, 45, 2.0, 1.0, split="none"))
        for c in case.boundary_conditions:
            if c.patch_name in ("left", "right"):
                c.kind, c.values = left if c.patch_name == "left" else right
            else:
                c.kind, c.mechanical_condition = "Wall", "Slip"
    g = build_geometry(case.mesh, case)
    n = len(g.areas)
    if kind in ("velocity", "total", "flow"):
        rng = np.random.default_rng(3)
        P = np.tile((1.0, 0.3, 0.0, 1.0), (n, 1)) + 0.02 * rng.standard_normal((n, 4))
    else:
        P = smooth_primitive(n, seed=2, amplitude=0.4)
    return case.numerics, g, P


@pytest.mark.parametrize("recon", ("MUSCL linear", "First order"))
@pytest.mark.parametrize("kind", tuple(SEGMENTS))
def test_flux_shapes_change_launches_and_no_bit(cuda_device, kind, recon):
    from meshcfd_gb300.device import DeviceGeometry, make_config, primitive_to_conservative

    s, g, P = _geometry(kind)
    s.reconstruction, s.limiter, s.flux = recon, "Venkatakrishnan", "HLLC"
    dg = DeviceGeometry(g)
    assert len(g.interior_faces) >= 152 * 32  # shapes of 32 threads apply
    U = torch.as_tensor(primitive_to_conservative(P, s.gamma), device=cuda_device)
    lib = dg.lib

    def residual(cfg, shapes):
        assert lib.mcfd_set_launch_shapes(dg.handle, (C.c_int32 * 5)(*shapes)) == 0
        before = lib.mcfd_launch_count()
        R = dg.residual(U, cfg)
        return lib.mcfd_launch_count() - before, R

    for mode in ("fast", "exact", "fma"):
        cfg = make_config(s, mode)
        launches, ref = residual(cfg, (0, 0, 0, 0, 0))
        dg.check_status()
        for threads, faces in ((32, 1), (32, 2), (32, 4), (32, 7), (64, 2), (256, 4)):
            n, R = residual(cfg, (0, threads, faces, 0, 0))
            apart = faces > 1 and len(g.interior_faces) >= 152 * threads
            assert n == launches + (SEGMENTS[kind] - 1 if apart else 0), (threads, faces)
            if mode == "fma":
                assert float((R - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
            else:
                assert torch.equal(R, ref), (mode, threads, faces)
    dg.check_status()
