"""Exterior states of pressure and mass-flow inlets, bit for bit: an exact-mode
residual of a duct whose inlet is a velocity inlet given the states that the
full bisections give (solver.py:4412-4577 restated in NumPy, the power by the
CUDA library's pow through PyTorch) equals the residual of the same duct with
the real inlet, on every cell.  Pressure inlets: Mach numbers from near
stagnation to near sonic, directions from normal to the inlet to almost along
it.  Mass-flow inlets: flow rates from next to none, patches around the
pairwise sum's leaves and around the 1,024 faces that fit shared memory.  And the viscosity of Sutherland's law in exact mode
by the same power, read back through the time steps."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

R_GAS, GAMMA = 287.05, 1.4


def _duct(ny, left):
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import box_mesh
    from meshcfd_gb300.model import Case

    case = Case(name="duct", mesh=box_mesh(2, ny, 2.0, 1.0, split="none"))
    for c in case.boundary_conditions:
        if c.patch_name == "left":
            c.kind, c.values = left
        elif c.patch_name == "right":
            c.kind, c.values = "Pressure Outlet", {"pressure": 0.9}
        else:
            c.kind, c.mechanical_condition = "Wall", "Slip"
    case.numerics.reconstruction = "First order"
    case.numerics.flux = "Rusanov"
    return case, build_geometry(case.mesh, case)


def _cuda_pow(x, y, device):
    """CUDA's pow, element by element."""
    x = torch.as_tensor(np.asarray(x, dtype=np.float64), device=device)
    return torch.pow(x, torch.full_like(x, y)).cpu().numpy()


def _residual(g, numerics, P, device, mode="exact"):
    from meshcfd_gb300.device import DeviceGeometry, make_config, primitive_to_conservative

    dg = DeviceGeometry(g)
    U = torch.as_tensor(primitive_to_conservative(P, GAMMA), device=device)
    cfg = make_config(numerics, mode)
    R = dg.residual(U, cfg).cpu().numpy()
    dg.check_status()
    return R, dg.primitive(U, cfg).cpu().numpy()


def _with_states(ny, faces, states):
    """The duct with a velocity inlet of one given state per face."""
    case, g = _duct(ny, ("Velocity Inlet", {"density": 1.0, "temperature": 1.0 / R_GAS, "velocity_x": 0.3}))
    assert np.array_equal(np.asarray(g.velocity_inlet_faces), np.asarray(faces))
    g.velocity_inlet_states = np.ascontiguousarray(states)
    return case, g


def _check(ny, g, numerics, P, faces, states, device):
    R, _ = _residual(g, numerics, P, device)
    _, gv = _with_states(ny, faces, states)
    ref, _ = _residual(gv, numerics, P, device)
    own = np.asarray(g.owners)[faces]
    assert np.all(np.abs(ref[own]).max(axis=0) > 0.0)
    np.testing.assert_array_equal(R, ref)


MACHS = (1e-9, 1e-4, 0.01, 0.1, 0.3, 0.5, 0.8, 0.95, 0.999, 1.0 - 1e-9)


@pytest.mark.parametrize("vy", (0.0, 0.2, 3.0, 1e3, 1e6))
@pytest.mark.parametrize("ny", (1, 10, 143))
def test_pressure_inlet_states_bit_for_bit(cuda_device, ny, vy):
    pt, tt = 1.2, 1.1 / R_GAS
    case, g = _duct(ny, ("Pressure Inlet", {"pressure": pt, "temperature": tt, "velocity_x": 1.0, "velocity_y": vy}))
    (inlet,) = g.pressure_inlets
    faces, d = np.asarray(inlet.faces), np.asarray(inlet.direction, dtype=np.float64)
    own = np.asarray(g.owners)[faces]
    normal = np.asarray(g.face_normals).reshape(-1, 2)[faces]
    dn = normal[:, 0] * d[0] + normal[:, 1] * d[1]
    a0 = np.sqrt(GAMMA * R_GAS * tt)

    def invariant(m):
        ratio = 1.0 + 0.5 * (GAMMA - 1.0) * (m * m)
        return a0 / np.sqrt(ratio) * (dn * m + 2.0 / (GAMMA - 1.0))

    # interior states whose outgoing invariant is that of a Mach number
    rng = np.random.default_rng(ny)
    P = np.tile((1.0, 0.05, 0.0, 1.0), (len(g.areas), 1))
    P[:, 0] += 0.05 * rng.standard_normal(len(P))
    P[:, 2] += 0.02 * rng.standard_normal(len(P))
    m = np.resize(MACHS, ny) * (1.0 if ny < 11 else rng.uniform(0.9, 1.0, ny))
    if vy > 1e4:  # closer to stagnation the invariant is that of no flow to rounding
        m = np.maximum(m, 1e-4)
    sound = 0.5 * (GAMMA - 1.0) * (invariant(m) - (P[own, 1] * normal[:, 0] + P[own, 2] * normal[:, 1]))
    P[own, 3] = sound * sound * P[own, 0] / GAMMA
    _, Ph = _residual(g, case.numerics, P, cuda_device)  # accepted: the status is checked
    q = Ph[own]
    un = q[:, 1] * normal[:, 0] + q[:, 2] * normal[:, 1]
    outgoing = un + 2.0 * np.sqrt(GAMMA * q[:, 3] / q[:, 0]) / (GAMMA - 1.0)
    low, high = np.zeros(ny), np.ones(ny)
    for _ in range(64):
        mid = 0.5 * (low + high)
        above = invariant(mid) > outgoing
        low, high = np.where(above, mid, low), np.where(above, high, mid)
    m = 0.5 * (low + high)
    t = tt / (1.0 + 0.5 * (GAMMA - 1.0) * (m * m))
    p = pt * _cuda_pow(t / tt, GAMMA / (GAMMA - 1.0), cuda_device)
    speed = m * np.sqrt(GAMMA * R_GAS * t)
    states = np.column_stack((p / (R_GAS * t), speed * d[0], speed * d[1], p))
    _check(ny, g, case.numerics, P, faces, states, cuda_device)


@pytest.mark.parametrize("ny", (1, 7, 8, 9, 127, 129, 200, 700, 1023, 1024, 1025, 1100))
@pytest.mark.parametrize("mdot", (1e-6, 0.3, 0.9))
def test_mass_flow_inlet_states_bit_for_bit(cuda_device, ny, mdot):
    tt = 1.1 / R_GAS
    case, g = _duct(ny, ("Mass Flow Inlet", {"mass_flow": mdot, "temperature": tt, "velocity_x": 1.0,
                                             "velocity_y": -0.1}))
    (inlet,) = g.mass_flow_inlets
    faces, d = np.asarray(inlet.faces), np.asarray(inlet.direction, dtype=np.float64)
    own = np.asarray(g.owners)[faces]
    normal = np.asarray(g.face_normals).reshape(-1, 2)[faces]
    proj = -(normal[:, 0] * d[0] + normal[:, 1] * d[1])
    length = np.asarray(g.face_lengths)[faces]
    rng = np.random.default_rng(ny)
    P = np.tile((1.0, 0.3, 0.0, 1.0), (len(g.areas), 1)) + 0.04 * rng.standard_normal((len(g.areas), 4))
    _, Ph = _residual(g, case.numerics, P, cuda_device)
    p = Ph[own, 3]
    cp = GAMMA * R_GAS / (GAMMA - 1.0)

    def below(s):
        rt = R_GAS * (tt - s * s / (2.0 * cp))
        return float(np.sum(p / rt * s * proj * length)) < mdot

    low, high = 0.0, np.sqrt(2.0 * cp * tt) * (1.0 - 1e-12)
    assert not below(high)
    for _ in range(80):
        mid = 0.5 * (low + high)
        low, high = (mid, high) if below(mid) else (low, mid)
    s = 0.5 * (low + high)
    rho = p / (R_GAS * (tt - s * s / (2.0 * cp)))
    states = np.column_stack((rho, np.full(ny, s * d[0]), np.full(ny, s * d[1]), p))
    _check(ny, g, case.numerics, P, faces, states, cuda_device)


@pytest.mark.parametrize("model", ("Constant", "Sutherland"))
def test_sutherland_viscosity_bit_for_bit(cuda_device, monkeypatch, model):
    import oracle.viscous
    from meshcfd_gb300.device import DeviceGeometry, make_config, primitive_to_conservative
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import periodic_case
    from oracle.oracle import Oracle

    case = periodic_case(24, 17, split="none", jitter=0.1, seed=3)
    s = case.numerics
    s.viscosity_model, s.dynamic_viscosity = model, 0.3
    s.sutherland_reference_viscosity, s.sutherland_reference_temperature = 0.4, 1.0 / R_GAS
    s.sutherland_temperature = 0.4 / R_GAS
    g = build_geometry(case.mesh, case)
    rng = np.random.default_rng(2)
    n = len(g.areas)
    P = np.tile((1.0, 0.3, 0.1, 1.0), (n, 1)) * (1.0 + 0.2 * rng.uniform(-1.0, 1.0, (n, 4)))
    dg, orc = DeviceGeometry(g), Oracle(g)
    cfg = make_config(s, "exact")
    Pd = dg.primitive(torch.as_tensor(primitive_to_conservative(P, GAMMA), device=cuda_device), cfg)
    dt, _ = dg.time_steps(Pd, cfg, per_cell=True)
    dg.check_status()

    def viscosity(T, s):
        if model == "Constant":
            return np.full_like(T, s.dynamic_viscosity)
        tref = s.sutherland_reference_temperature
        mu = s.sutherland_reference_viscosity * _cuda_pow(T / tref, 1.5, cuda_device)
        return mu * ((tref + s.sutherland_temperature) / (T + s.sutherland_temperature))

    monkeypatch.setattr(oracle.viscous, "dynamic_viscosity", viscosity)
    np.testing.assert_array_equal(dt.cpu().numpy(), orc.stable_time_steps(Pd.cpu().numpy(), s))
