"""The time step's far-field radius from the characteristic sound speed (fast
mode) and its hand-over to the whole far-field state, against the oracle.

Both routes hold the same value up to the rounding of three powers (exponents
up to 2.5), two quotients and a root: under 20 units of 1.1e-16 in the radius,
and the cell's sum and quotient add under ten, so 1e-14 bounds the step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(kind, P, rng):
    P = P * (1.0 + 0.05 * rng.standard_normal(P.shape))
    if kind == "supersonic":
        P[:, 1:3] *= rng.uniform(1.0, 8.0, (len(P), 1))
    elif kind == "reversed":  # inflow where the free stream leaves
        P[:, 1:3] *= -1.0
    elif kind == "thin":  # density and pressure beyond the short route's range
        P[:, [0, 3]] *= 10.0 ** rng.uniform(-60, 60, (len(P), 1))
    elif kind == "hot":  # sound speeds far from the free stream's
        P[:, 3] *= 10.0 ** rng.uniform(-3, 3, len(P))
    return np.ascontiguousarray(P)


@pytest.mark.parametrize("mesh", ("bump", "ogrid"))
@pytest.mark.parametrize("kind", ("ordinary", "supersonic", "reversed", "thin", "hot"))
def test_local_time_steps_with_far_field(cuda_device, mesh, kind):
    import torch
    from meshcfd_gb300.device import DeviceGeometry, make_config
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import bump_case, ogrid_case
    from oracle.oracle import Oracle

    case, P = bump_case(40, 24) if mesh == "bump" else ogrid_case(64, 20)
    P = states(kind, P, np.random.default_rng(11))
    g = build_geometry(case.mesh, case)
    dg = DeviceGeometry(g)
    got = dg.time_steps(torch.as_tensor(P, device=cuda_device), make_config(case.numerics, "fast"), per_cell=True)[0]
    dg.check_status()
    ref = Oracle(g).stable_time_steps(P, case.numerics)
    np.testing.assert_allclose(got.cpu().numpy(), ref, rtol=1e-14)
