"""Support radii at which fluid at rest has more neighbours than a kept list holds (512, from about 4.9 r on): the
oracle's bits, scenes without iterations among others in a batch, and little time lost on lists that overflow."""
import time

import numpy as np
import pytest

from novaphy_gb300 import capi
from test_gpu_walk_forms import block, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_factor", [4.8, 5.0, 6.0])
def test_bits(port_mt, h_factor):
    check(port_mt, block(140000, h_factor=h_factor, seed=23, vorticity=1e-4), 2)


def test_scenes_without_iterations(port_mt):
    # Their velocity passes list for the first time in the step, whatever the lists of the step before were.
    from oracle.oracle import Settings

    ws = [block(70000, h_factor=6.0, seed=24), block(70000, h_factor=6.0, seed=25), block(9000, h_factor=4.0, seed=26)]
    iters = (2, 0, 1)
    b, scs = capi.Batch(), []
    for w, it in zip(ws, iters):
        w.settings["solver_iterations"] = it
        sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
        sc.set_gravity(w.gravity)
        scs.append(sc)
    b.step(scs, [w.dt for w in ws], [2] * len(ws))
    b.sync()
    for sc, w in zip(scs, ws):
        z = np.zeros(w.n, np.float32)
        want = port_mt.steps(Settings.make(**w.settings), w.x, w.v, z, z, w.dt, w.gravity, w.mass, 2)
        for name, p, q in zip("x v rho lam".split(), sc.state(), want):
            assert np.array_equal(p, q), name
    for o in scs + [b]:
        o.close()


@pytest.mark.parametrize("h_factor", [4.8, 5.0, 5.3])
def test_same_bits_over_steps_that_list_and_steps_that_do_not(h_factor):
    # 31 steps without lists follow one whose lists overflowed.
    w = block(140000, h_factor=h_factor, seed=28, vorticity=1e-4)
    out = []
    for on in (True, False):
        sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=1), w.x, w.v, mass=w.mass)
        sc.set_gravity(w.gravity)
        sc.set_kept_lists(on)
        sc.step(w.dt, 70)
        out.append([a.view(np.uint32) for a in sc.state()])
        sc.close()
    assert all(np.array_equal(p, q) for p, q in zip(*out))


def test_time_of_lists_that_overflow():
    # Five listings that overflow cost a third of a step that walks; one costs a fifth of that.
    w = block(262144, h_factor=6.0, seed=27, vorticity=1e-4)
    best = {}
    for on in (True, False):
        sc = capi.Scene(capi.default_settings(**w.settings), w.x, w.v, mass=w.mass)
        sc.set_gravity(w.gravity)
        sc.set_kept_lists(on)
        snap, t = sc.snapshot(), []
        for _ in range(6):
            sc.restore(snap)
            sc.sync()
            t0 = time.perf_counter()
            sc.step(w.dt)
            sc.sync()
            t.append(time.perf_counter() - t0)
        best[on] = min(t)
        snap.close()
        sc.close()
    assert best[True] < 1.2 * best[False], best
