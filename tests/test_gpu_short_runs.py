"""Runs of identical particles in ranges of fewer than 1,024 candidates next to a pile whose runs are summed as one
(large scenes): every particle counts once, whichever way its range is walked.  The oracle's bits, with and without
kept lists."""
import numpy as np
import pytest

from novaphy_gb300 import capi
from test_gpu_walk_forms import block

pytestmark = pytest.mark.gpu


def with_piles(n, origin):
    """n particles; a pile with a run of 1,500 in one cell, runs of 2 to 60 in the cells around it."""
    w = block(n, seed=31, vorticity=1e-4)
    rng = np.random.default_rng(33)
    h = w.settings["kernel_radius"]
    if origin:  # cells on both sides of the axes share reference keys
        w.x = (w.x - w.x.mean(0)).astype(np.float32)
        half = tuple(0.75 * t for t in w.settings["domain_upper"])
        w.settings.update(domain_lower=tuple(-t for t in half), domain_upper=half)
    cell = np.array([0, 0, 0] if origin else [8, 7, 9])
    at = lambda c: (np.asarray(c) + 0.2 + 0.6 * rng.random(3)) * h  # noqa: E731
    groups = [(at(cell), 1500)]
    for k, d in enumerate([(1, 0, 0), (0, 1, 0), (0, -1, 0), (1, 1, 0), (0, 0, 1), (-1, 0, -1), (1, -1, 1), (0, 1, -1)]):
        groups += [(at(cell + d), m) for m in (2 + k, 60 - k)]
    i = np.arange(5000, n)  # next to each other in the index, so that they are in cell order
    for x, m in groups:
        w.x[i[:m]], w.v[i[:m]] = x.astype(np.float32), 0.0
        i = i[m:]
    return w


@pytest.mark.parametrize("lists", [True, False])
@pytest.mark.parametrize("origin", [False, True])
def test_bits(port_mt, lists, origin):
    from oracle.oracle import Settings

    w = with_piles(140000, origin)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.set_kept_lists(lists)
    sc.step(w.dt)
    got = sc.state()
    sc.close()
    z = np.zeros(w.n, np.float32)
    want = port_mt.steps(Settings.make(**w.settings), w.x, w.v, z, z, w.dt, w.gravity, w.mass, 1)
    for name, a, b in zip("x v rho lam".split(), got, want):
        bad = np.flatnonzero(~((a == b) | (np.isnan(a) & np.isnan(b))).reshape(len(a), -1).all(1))
        assert bad.size == 0, (name, bad[:5], bad.size)
