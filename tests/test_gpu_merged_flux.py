"""Face fluxes in one launch (up to 500,000 faces) and in one launch per
segment (above): residuals on either side of the line, with walls and far
field, against the oracle (far field within the last places of its powers,
as in the other parity tests), and on the smallest meshes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("n", (1, 2, 5, 400, 410))  # 5, 16, 85, 480,800 and 505,120 faces
@pytest.mark.parametrize("flux", ("Rusanov", "HLLC", "Roe"))
def test_merged_and_separate_segments_match_the_oracle(cuda_device, n, flux):
    import torch
    from meshcfd_gb300.device import DeviceGeometry, make_config
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import riemann_case, smooth_primitive
    from oracle.oracle import Oracle

    case, P = riemann_case(n)
    s = case.numerics
    s.flux, s.reconstruction, s.limiter = flux, "MUSCL linear", "Minmod"
    g = build_geometry(case.mesh, case)
    assert len(g.face_lengths) == 3 * n * n + 2 * n
    orc = Oracle(g)
    U = orc.conservative(smooth_primitive(len(P), seed=2, amplitude=0.4), s.gamma)
    dg = DeviceGeometry(g)
    for mode in ("fast", "exact"):
        R = dg.residual(torch.as_tensor(U, device=cuda_device), make_config(s, mode)).cpu().numpy()
        dg.check_status()
        assert rel_err(R, orc.residual(U, s)) <= 1e-15, mode
