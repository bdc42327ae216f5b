"""The default LU-SGS sweep (the pipelined band sweep where it can be
planned) against the one-block sweep with a barrier per level, bit for bit:
meshes smaller than the cluster, bands of less than a mesh row, steps of one
and of two groups of rows, a self-coupled periodic row, triangles, cells of
five and six faces and random numbering (which take another schedule), after
repeated applications and after the schedule was chosen with the operator
already prepared."""

import numpy as np
import pytest

from test_gpu_implicit import _permuted_periodic, _prepare_on

pytestmark = pytest.mark.gpu


def _mesh(kind):
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import bump_case, periodic_case
    from test_gpu_polygons import _polygon_case

    if kind == "polygons":
        case = _polygon_case()
    elif kind == "permuted":
        return _permuted_periodic(64, 3)
    elif kind[0] == "bump":
        case = bump_case(kind[1], kind[2])[0]
    else:
        case = periodic_case(kind[1], kind[2], split=kind[0], jitter=0.1 if min(kind[1:]) > 2 else 0.0, seed=6)
    s = case.numerics
    s.time_step_mode = "Local (steady)"
    s.cfl = 20.0
    return case, build_geometry(case.mesh, case)


@pytest.mark.parametrize("kind", (("none", 1, 1), ("none", 3, 1), ("bump", 3, 2), ("bump", 17, 5), ("bump", 64, 33),
                                  ("bump", 301, 149), ("bump", 128, 272), ("all", 61, 25), ("half", 90, 70),
                                  "polygons", "permuted"))
def test_default_sweep_equals_the_barrier_sweep(cuda_device, kind):
    import torch
    from meshcfd_gb300.meshes import smooth_primitive

    case, g = _mesh(kind)
    P = smooth_primitive(len(g.areas), seed=8, amplitude=0.5)
    dg, U0, _, _ = _prepare_on(g, case.numerics, P, cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(1)
    vs = [torch.as_tensor(rng.standard_normal(U0.shape), device=cuda_device) for _ in range(3)]

    def apply_all():
        out = []
        for v in vs:
            x = torch.empty_like(v)
            assert dg.lib.mcfd_lusgs_apply(dg.handle, v.data_ptr(), x.data_ptr(), stream) == 0
            out.append(x)
        return [x.cpu().numpy() for x in out]

    first = apply_all()
    assert dg.lib.mcfd_implicit_set_sweep(dg.handle, 0, 1) == 0
    barrier = apply_all()
    assert dg.lib.mcfd_implicit_set_sweep(dg.handle, 0, 0) == 0
    again = apply_all()
    dg.check_status()
    for a, b, c in zip(first, barrier, again):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(c, b)
