"""Coupling sums over values that are not finite, against the oracle: a position, density or volume that is
not a number or infinite spoils the sums of the points whose buckets hold it, as in the reference, and no others;
forces that are not numbers stay off the bodies."""
import numpy as np
import pytest

from novaphy_gb300 import capi, workloads
from test_gpu_coupling import port_coupling_accumulated

pytestmark = pytest.mark.gpu

BAD = [np.nan, np.inf, -np.inf]


def put(a, at, value):
    a[at] = value
    return a


@pytest.mark.parametrize("spacing", [0.02, 0.004])  # teams of 8 and of 16
@pytest.mark.parametrize("value", BAD)
def test_volumes(port_mt, spacing, value):
    # A value that is not a number falls into cell 0: the samples lie around the origin.
    pts = port_mt.sample_box([0.12, 0.1, 0.11], (0, 0, 0), [1, 0, 0, 0], np.float32(spacing)).astype(np.float32)
    for at in (5, len(pts) // 2):
        w = put(pts.copy(), (at, at % 3), value)
        if value == np.inf:
            w[at + 7] = w[at]  # two at infinity are no number apart
        got, want = capi.boundary_volumes(w, np.float32(0.05)), port_mt.boundary_volumes(w, np.float32(0.05))
        assert np.array_equal(got, want), np.flatnonzero(got != want)[:5]


def world(port, edge, spacing):
    w = workloads.dam_break((edge,) * 3, 0.025, (1.5, 1.5, 1.5), dt=1.0 / 120.0, seed=edge, vorticity=0.0)
    w.x = (w.x * np.float32(0.9)).astype(np.float32)
    ident = np.array([1, 0, 0, 0], np.float32)
    parts = [port.sample_sphere(0.07, (0, 0, 0), ident, np.float32(spacing)),
             port.sample_box([0.05, 0.05, 0.05], (0, 0, 0), ident, np.float32(spacing))]
    local = np.concatenate(parts).astype(np.float32)
    body = np.repeat([0, 1], [len(p) for p in parts]).astype(np.int32)
    pos = np.array([[0.08, 0.09, 0.07], [0.14, 0.05, 0.16]], np.float32)
    return w, local, body, pos, np.stack([ident, ident]).astype(np.float32)


@pytest.mark.parametrize("edge,spacing", [(9, 0.02), (22, 0.005)])
@pytest.mark.parametrize("where", ["x", "rho", "psi", "none"])
@pytest.mark.parametrize("value", BAD)
def test_coupling(port_mt, edge, spacing, where, value):
    port = port_mt
    w, local, body, pos, quat = world(port, edge, spacing)
    h = np.float32(w.settings["kernel_radius"])
    dyn = np.array([1, 1], np.int32)
    world0 = port.boundary_world_positions(local, body, pos, quat)
    psi = port.boundary_volumes(world0, h)
    if where == "psi":
        psi[len(psi) // 3] = value
    z = np.zeros((2, 3), np.float32)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.set_boundary(local, body, psi)
    sc.set_bodies(pos, quat, dyn)
    sc.step(w.dt, 1)
    x, _, rho, _ = sc.state()
    near = np.argsort(((x - pos[0]) ** 2).sum(1))
    if where == "x":
        x[near[3], 1] = value
        x[near[40]] = value
    if where == "rho":
        rho[near[[3, 200]]] = value
    sc.write(capi.FIELD_POSITIONS, x)
    sc.write(capi.FIELD_DENSITIES, rho)
    f, t = sc.couple(w.dt, z, z)
    got = sc.state()[2]
    sc.close()
    want = port.boundary_density(x, rho, world0, psi, h, np.float32(1000.0))
    assert np.array_equal(got, want, equal_nan=True), np.flatnonzero(~((got == want) | (got != got)))[:5]
    wf, wt = port_coupling_accumulated(port, x, want, w.mass, world0, body, psi, dyn, pos, h, z, z)
    assert np.array_equal(f, wf, equal_nan=True) and np.array_equal(t, wt, equal_nan=True)
