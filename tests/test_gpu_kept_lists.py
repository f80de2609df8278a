"""The candidate lists that the density pass keeps for the delta pass, and the XSPH pass for the vorticity pass,
against the oracle, bit for bit: piles of as many particles as a list has room for and a few more and fewer,
several iterations (particles that nothing moved around keep an earlier iteration's list), runs of identical
particles, whose lists are not kept, and a batch of scenes that end after different numbers of iterations."""
import numpy as np
import pytest

from novaphy_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def scene(n, pile, seed=0, same=False, r=0.02, **kw):
    """A lattice of n particles in the lower half of a box; `pile` of them in one cell of the upper half."""
    e = int(np.ceil(n ** (1.0 / 3.0)))
    w = workloads.dam_break((e, e, e), r, (2.0 * e * r + 16 * r,) * 3, jitter=0.05 * r, seed=seed, **kw)
    rng = np.random.default_rng(seed + 1)
    w.x = w.x[:n].copy()
    w.v = (rng.normal(size=w.x.shape) * 0.2).astype(np.float32)
    at = rng.permutation(n)[:pile]
    spread = np.zeros((pile, 3)) if same else 0.2 * rng.random((pile, 3))
    w.x[at] = ((2.0 * e + 10 + spread) * r).astype(np.float32)
    w.v[at] = 0.0
    return w


def oracle_of(port_mt, w, nsteps):
    from oracle.oracle import Settings

    z = np.zeros(w.n, np.float32)
    return port_mt.steps(Settings.make(**w.settings), w.x, w.v, z, z, w.dt, w.gravity, w.mass, nsteps)


def same_bits(got, want):
    for name, a, b in zip("x v rho lam".split(), got, want):
        assert np.array_equal(a, b, equal_nan=True), name


@pytest.mark.parametrize("n", [3000, 40000, 140000])
@pytest.mark.parametrize("pile", [510, 511, 512, 513, 1025])
def test_room(port_mt, n, pile):
    w = scene(n, pile, seed=pile, vorticity=1e-4)
    w.settings.update(corr_k=0.001, corr_delta_q=0.3)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.step(w.dt, 2)
    same_bits(sc.state(), oracle_of(port_mt, w, 2))
    sc.close()


@pytest.mark.parametrize("n", [3000, 140000])
def test_identical_particles(port_mt, n):
    w = scene(n, 1200, seed=3, same=True, vorticity=1e-4)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.step(w.dt, 1)
    same_bits(sc.state(), oracle_of(port_mt, w, 1))
    sc.close()


@pytest.mark.parametrize("sizes", [(700, 1, 1300), (60000, 45000, 40000)])
def test_batch_of_different_iterations(port_mt, sizes):
    ws = [scene(n, min(n, 513), seed=k, vorticity=1e-4 if k == 1 else 0.0, iterations=2 + k)
          for k, n in enumerate(sizes)]
    scs = [capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass) for w in ws]
    for sc, w in zip(scs, ws):
        sc.set_gravity(w.gravity)
    b = capi.Batch()
    b.step(scs, [w.dt for w in ws], [2] * len(ws))
    for sc, w in zip(scs, ws):
        same_bits(sc.state(), oracle_of(port_mt, w, 2))
        sc.close()
    b.close()
