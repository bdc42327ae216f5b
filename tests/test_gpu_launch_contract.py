"""What a launch-shape call leaves behind: zeros restore the default shapes,
and a tuning under any mode, limiter or reconstruction keeps the
reconstruction's default form (one thread per (cell, variable)), reports it,
and can be replayed from its report.  In fma mode the forms of the
reconstruction would contract differently, so the bits there follow the form."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _vortex(n, limiter, recon):
    from meshcfd_gb300.device import primitive_to_conservative
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import cell_centroids, vortex_case, vortex_primitive

    case, _ = vortex_case(n, split="half")
    s = case.numerics
    s.limiter, s.reconstruction = limiter, recon
    P = vortex_primitive(cell_centroids(case.mesh))
    P *= 1.0 + 0.01 * np.random.default_rng(4).standard_normal(P.shape)
    return s, build_geometry(case.mesh, case), primitive_to_conservative(P, s.gamma)


def _set(dg, shapes):
    assert dg.lib.mcfd_set_launch_shapes(dg.handle, (C.c_int32 * 5)(*shapes)) == 0


@pytest.mark.parametrize("mode,limiter,recon", (
    ("exact", "Venkatakrishnan", "MUSCL linear"), ("fma", "Van Leer", "MUSCL linear"),
    ("fast", "Minmod", "MUSCL linear"), ("fast", "Venkatakrishnan K", "MUSCL linear"),
    ("fast", "Minmod", "First order")))
def test_tuning_keeps_the_default_reconstruction(cuda_device, mode, limiter, recon):
    from meshcfd_gb300.device import DeviceGeometry, make_config

    s, g, U = _vortex(24, limiter, recon)
    U = torch.as_tensor(U, device=cuda_device)
    cfg = make_config(s, mode)
    dg = DeviceGeometry(g)
    fma = make_config(s, "fma")
    before = dg.residual(U, cfg).clone(), dg.residual(U, fma).clone()
    chosen = dg.autotune(U, cfg)
    assert chosen["reconstruct_per_variable"] == 1
    for shapes in (None, list(chosen.values()), (0, 0, 0, 0, 0)):
        if shapes:
            _set(dg, shapes)
        assert torch.equal(dg.residual(U, cfg), before[0])
        assert torch.equal(dg.residual(U, fma), before[1])
    dg.check_status()
