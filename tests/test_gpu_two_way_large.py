"""Two-way coupling in scenes of more than 131,072 particles, where some warps read kept lists and others (a pile of
more candidates than a list holds, thrown particles) walk: each warp adds the boundary's share once.  Boundary volumes
of zero give the one-way step's bits, and real ones the same bits with and without lists."""
import numpy as np
import pytest

from novaphy_gb300 import capi
from test_gpu_walk_forms import block

pytestmark = pytest.mark.gpu

IDENT = np.array([1, 0, 0, 0], np.float32)


def run(port, lists, two_way, psi_scale, friction=0.0, nsteps=2):
    w = block(140000, seed=41)
    w.settings.update(corr_k=0.001, corr_delta_q=0.3, vorticity_epsilon=1e-4 if friction else 0.0)
    rng = np.random.default_rng(43)
    pick = rng.permutation(w.n)
    pile, far = pick[:1400], pick[1400:1700]
    w.x[pile] = (0.55 + 0.01 * rng.random((1400, 3))).astype(np.float32)
    w.v[pile] = 0.0
    w.v[far] *= np.float32(10.0 * w.settings["kernel_radius"] / w.dt)
    h = np.float32(w.settings["kernel_radius"])
    pos = np.array([[0.5, 0.45, 0.4], [0.3, 0.3, 0.9]], np.float32)
    quat = np.stack([IDENT, IDENT])
    parts = [port.sample_box([0.15, 0.12, 0.1], (0, 0, 0), IDENT, np.float32(0.02)),
             port.sample_sphere(0.1, (0, 0, 0), IDENT, np.float32(0.02))]
    local = np.concatenate(parts).astype(np.float32)
    body = np.repeat([0, 1], [len(p) for p in parts]).astype(np.int32)
    psi = port.boundary_volumes(port.boundary_world_positions(local, body, pos, quat), h) * np.float32(psi_scale)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1, boundary_two_way=two_way,
                                          boundary_friction=friction), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.set_kept_lists(lists)
    sc.set_boundary(local, body, psi.astype(np.float32))
    sc.set_bodies(pos, quat, np.array([1, 1], np.int32))
    z = np.zeros((2, 3), np.float32)
    out = []
    for _ in range(nsteps):
        out += sc.step_coupled(w.dt, z, z)
    out += sc.state()
    sc.close()
    return [np.ascontiguousarray(a).view(np.uint32) for a in out]


def same(a, b):
    return all(np.array_equal(p, q) for p, q in zip(a, b))


@pytest.mark.parametrize("lists", [True, False])
def test_zero_volumes_equal_one_way(port_mt, lists):
    assert same(run(port_mt, lists, 1, 0.0), run(port_mt, lists, 0, 0.0))


@pytest.mark.parametrize("friction", [0.0, 0.4])
def test_same_bits_with_and_without_lists(port_mt, friction):
    with_lists = run(port_mt, True, 1, 1.0, friction)
    assert same(with_lists, run(port_mt, False, 1, 1.0, friction))
    assert not same(with_lists, run(port_mt, True, 0, 1.0, friction))
