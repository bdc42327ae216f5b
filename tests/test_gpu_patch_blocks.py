"""Boundary-state patches of many sizes in one geometry (a block per 128 faces
of a patch, 64 at most): the residual of a batch equals those of its cases, bit
for bit, for patches from 1 face to more than 64 blocks take at a face a thread."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

R_GAS = 287.05
VELOCITY = ("Velocity Inlet", {"density": 1.0, "temperature": 1.0 / R_GAS, "velocity_x": 0.3, "velocity_y": 0.0})
TOTAL = ("Pressure Inlet", {"pressure": 1.2, "temperature": 1.1 / R_GAS, "velocity_x": 1.0, "velocity_y": 0.1})
FLOW_IN = ("Mass Flow Inlet", {"mass_flow": 0.3, "temperature": 1.1 / R_GAS, "velocity_x": 1.0, "velocity_y": 0.0})
FLOW_OUT = ("Mass Flow Outlet", {"mass_flow": 0.3})
STATIC = ("Pressure Outlet", {"pressure": 0.9})


def _duct(ny, left, right):
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import box_mesh
    from meshcfd_gb300.model import Case

    case = Case(name="duct", mesh=box_mesh(2, ny, 2.0, 1.0, split="none"))
    for c in case.boundary_conditions:
        if c.patch_name in ("left", "right"):
            c.kind, c.values = left if c.patch_name == "left" else right
        else:
            c.kind, c.mechanical_condition = "Wall", "Slip"
    s = case.numerics
    s.flux, s.reconstruction = "HLLC", "First order"
    return s, build_geometry(case.mesh, case)


@pytest.mark.parametrize("mode", ("fast", "exact"))
def test_patches_of_many_sizes(cuda_device, mode):
    from meshcfd_gb300.batch import concatenate
    from meshcfd_gb300.device import DeviceGeometry, make_config, primitive_to_conservative

    cases = [(ny, left, right) for ny in (1, 127, 129, 400) for left, right in ((TOTAL, STATIC), (FLOW_IN, FLOW_OUT))]
    cases += [(64 * 128 + 5, TOTAL, FLOW_OUT), (257, VELOCITY, FLOW_OUT), (3, FLOW_IN, STATIC)]
    rng = np.random.default_rng(7)
    geoms, states, parts = [], [], []
    for ny, left, right in cases:
        s, g = _duct(ny, left, right)
        n = len(g.areas)
        P = np.tile((1.0, 0.3, 0.0, 1.0), (n, 1)) + 0.02 * rng.standard_normal((n, 4))
        U = primitive_to_conservative(P, s.gamma)
        dg = DeviceGeometry(g)
        parts.append(dg.residual(torch.as_tensor(U, device=cuda_device), make_config(s, mode)).cpu().numpy())
        dg.check_status()
        geoms.append(g)
        states.append(U)
    dg = DeviceGeometry(concatenate(geoms)[0])
    before = dg.lib.mcfd_launch_count()
    R = dg.residual(torch.as_tensor(np.concatenate(states), device=cuda_device), make_config(s, mode)).cpu().numpy()
    assert dg.lib.mcfd_launch_count() - before == 4  # primitive, states, fluxes, gather
    dg.check_status()
    np.testing.assert_array_equal(R, np.concatenate(parts))
