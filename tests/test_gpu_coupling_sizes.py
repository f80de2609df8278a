"""The coupling's sums at both team sizes (fewer and more than 8,192 boundary points or fluid particles), with
bodies of fewer and more points than one round of the per-body reduction, static bodies and world-owned points
between them, against the oracle bit for bit."""
import numpy as np
import pytest

from novaphy_gb300 import capi, workloads
from test_gpu_coupling import port_coupling_accumulated, quat_z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge,spacing,extent", [(9, 0.025, 0.4), (24, 0.025, 0.8), (13, 0.006, 0.3)])
def test_coupled_step_sizes(port_mt, edge, spacing, extent):
    from oracle.oracle import Settings

    port = port_mt
    w = workloads.dam_break((edge, edge + 1, edge), 0.025, (1.5, 1.5, 1.5), dt=1.0 / 120.0, seed=edge, vorticity=0.0)
    w.x = (w.x * np.float32(0.9)).astype(np.float32)  # denser than rest: pressure everywhere
    h, sp = np.float32(w.settings["kernel_radius"]), np.float32(spacing)
    ident = np.array([1, 0, 0, 0], np.float32)
    parts = [(port.sample_sphere(0.07, (0, 0, 0), ident, sp), 0),
             (port.sample_plane([0, 0, 1], 0.0, sp, extent), -1),
             (port.sample_box([0.06, 0.05, 0.04], (0, 0, 0), ident, sp), 1),
             (port.sample_sphere(0.03, (0, 0, 0), ident, sp), 2)]
    local = np.concatenate([p for p, _ in parts]).astype(np.float32)
    body = np.concatenate([np.full(len(p), k) for p, k in parts]).astype(np.int32)
    mid = 0.5 * 0.9 * edge * 0.025
    pos = np.array([[mid, mid, mid], [1.5 * mid, mid, 0.1], [0.05, 0.05, mid]], np.float32)
    quat = np.stack([quat_z(20.0), quat_z(30.0), ident]).astype(np.float32)
    dyn = np.array([1, 0, 1], np.int32)
    world0 = port.boundary_world_positions(local, body, pos, quat)
    psi = capi.boundary_volumes(world0, h)
    assert np.array_equal(psi, port.boundary_volumes(world0, h))
    f0 = np.array([[0.1, -0.2, -0.0], [0.0, 0.0, 0.0], [-0.0, 0.0, 1.0]], np.float32)
    t0 = np.array([[0.01, -0.0, -0.03], [0.0, 0.0, 0.0], [0.0, 2.0, -0.0]], np.float32)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.set_boundary(local, body, psi)
    sc.set_bodies(pos, quat, dyn)
    f, t = sc.step_coupled(w.dt, f0, t0)
    x, v, rho, lam = sc.state()
    sc.close()
    z = np.zeros(w.n, np.float32)
    ox, ov, orho, olam = port.steps(Settings.make(**w.settings), w.x, w.v, z, z, w.dt, w.gravity, w.mass, 1)
    orho = port.boundary_density(ox, orho, world0, psi, h, np.float32(1000.0))
    assert np.array_equal(x, ox) and np.array_equal(lam, olam) and np.array_equal(rho, orho)
    want_f, want_t = port_coupling_accumulated(port, ox, orho, w.mass, world0, body, psi, dyn, pos, h, f0, t0)
    assert np.array_equal(f.view(np.uint32), want_f.view(np.uint32))
    assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))
