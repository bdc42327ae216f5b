"""The parabolic reconstruction's mesh-only plan and its per-variable kernel at
their edges: cell counts around the block size of four threads per cell,
cells with 5 and 6 limiter entries, a one-row strip whose stencils are all
rank deficient, and the fields entry point — bit for bit against the oracle
(the kernel keeps its operation order)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITERS = ("Barth-Jespersen", "Minmod", "Van Leer", "Venkatakrishnan")


def _case(kind):
    from meshcfd_gb300.meshes import periodic_case
    from test_gpu_polygons import _polygon_case

    if kind == "polygons":
        return _polygon_case()
    nx, ny, split = kind
    return periodic_case(nx, ny, split=split, jitter=0.2 if min(nx, ny) > 2 else 0.0, seed=4)


@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("kind", ("polygons", (31, 1, "none"), (4, 4, "none"), (11, 3, "none"), (8, 4, "none"),
                                  (9, 7, "half"), (16, 8, "all")))
def test_plan_and_per_variable_kernel_match_the_oracle(cuda_device, kind, limiter):
    import torch
    from meshcfd_gb300.device import DeviceGeometry, make_config
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import smooth_primitive
    from oracle.oracle import Oracle

    case = _case(kind)
    s = case.numerics
    s.flux, s.reconstruction, s.limiter = "HLLC", "MUSCL parabolic", limiter
    g = build_geometry(case.mesh, case)
    assert len(g.parabolic_sources) > 0
    orc = Oracle(g)
    U = orc.conservative(smooth_primitive(len(g.areas), seed=9, amplitude=0.5), s.gamma)
    dg = DeviceGeometry(g)
    cfg = make_config(s)
    Ud = torch.as_tensor(U, device=cuda_device)
    np.testing.assert_array_equal(dg.residual(Ud, cfg).cpu().numpy(), orc.residual(U, s))
    P = orc.primitive(U, s.gamma)
    for a, b in zip(dg.reconstruction(torch.as_tensor(P, device=cuda_device), cfg),
                    orc.parabolic_reconstruction(P, limiter)):
        np.testing.assert_array_equal(a.cpu().numpy(), b)
    dg.check_status()
