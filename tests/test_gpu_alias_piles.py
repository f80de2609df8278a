"""Piles whose slot also holds particles from outside the grid box: runs of several cells alternate within the slot,
and cells share reference keys (merged buckets).  Bits of the oracle, and a neighbour structure whose time does not
grow with the square of the pile."""
import numpy as np
import pytest

from novaphy_gb300 import capi

pytestmark = pytest.mark.gpu

H, DT = 0.1, 0.01


def ref_key(c):
    c = np.asarray(c, np.int64).astype(np.uint64)
    return (c[..., 0] * np.uint64(73856093)) ^ (c[..., 1] * np.uint64(19349663)) ^ (c[..., 2] * np.uint64(83492791))


def shared_key_cells():
    """Two cells within [-3, 3)^3 with one reference key."""
    cells = np.stack(np.meshgrid(*[np.arange(-3, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    keys = ref_key(cells)
    order = np.argsort(keys, kind="stable")
    k = np.flatnonzero(keys[order][1:] == keys[order][:-1])[0]
    return cells[order[k]], cells[order[k + 1]]


def pile(n, pattern, seed=0):
    """n particles: A (a cell), B (a cell one grid period away, in A's slot) and C (a cell with A's key), in the order
    of the pattern.  The box is [-0.55, 0.55]^3, so the grid is 12 + 4 cells wide."""
    rng = np.random.default_rng(seed)
    a, c = shared_key_cells()
    if pattern == "stray":
        kind = np.zeros(n, int)
        kind[n // 2] = 1
    elif pattern == "turn":
        kind = np.arange(n) % 2
    elif pattern == "stray_merged":
        kind = np.arange(n) % 2 * 2
        kind[[n // 3, n // 2]] = 1
    else:
        kind = rng.integers(0, 3, n)
    at = np.stack([a, a, c])[kind]
    x = ((at + 0.1 + 0.8 * rng.random((n, 3))) * H).astype(np.float32)
    v = np.zeros((n, 3), np.float32)
    v[kind == 1, 0] = 16 * H / DT
    return x, v


SETTINGS = dict(kernel_radius=H, use_domain_bounds=1, domain_lower=(-0.55,) * 3, domain_upper=(0.55,) * 3,
                solver_iterations=2, particle_radius=0.025)
G = np.zeros(3, np.float32)
MASS = np.float32(0.125)


def scene(x, v, **kw):
    sc = capi.Scene(capi.default_settings(**SETTINGS, exact_arithmetic=1, **kw), x, v, mass=MASS)
    sc.set_gravity(G)
    return sc


def oracle(port_mt, x, v):
    from oracle.oracle import Settings

    z = np.zeros(len(x), np.float32)
    return port_mt.steps(Settings.make(**SETTINGS), x, v, z, z, np.float32(DT), G, MASS, 1)


# Fewer and more than a round of the cooperative scans.
@pytest.mark.parametrize("n", [5, 127, 128, 129, 260, 3001])
@pytest.mark.parametrize("pattern", ["stray", "turn", "stray_merged", "three"])
def test_bits(port_mt, n, pattern):
    x, v = pile(n, pattern, seed=n)
    sc = scene(x, v)
    sc.step(DT)
    got = sc.state()
    sc.close()
    for name, p, q in zip("x v rho lam".split(), got, oracle(port_mt, x, v)):
        assert np.array_equal(p, q), (name, np.flatnonzero(~(p == q).reshape(n, -1).all(1))[:5])


def test_bits_in_a_batch(port_mt):
    states = [pile(n, p, seed=n) for n, p in ((400, "three"), (1, "stray"), (300, "turn"), (700, "stray_merged"))]
    scs, b = [scene(x, v) for x, v in states], capi.Batch()
    b.step(scs, [DT] * len(scs), [1] * len(scs))
    b.sync()
    for sc, (x, v) in zip(scs, states):
        for p, q in zip(sc.state(), oracle(port_mt, x, v)):
            assert np.array_equal(p, q)
    for o in scs + [b]:
        o.close()


@pytest.mark.parametrize("pattern", ["turn", "stray_merged", "three"])
def test_time_of_the_structure(pattern):
    # A warp takes 60,000 positions in 470 rounds, three times a cell, at 2 us a round for the loads: 3 ms for the
    # cells side by side.  30,000 dependent loads of 0.6 us, one thread's way along the runs, are 18 ms.
    x, v = pile(60000, pattern)
    sc = scene(x, v)
    ms = []
    snap = sc.snapshot()
    for _ in range(3):
        sc.restore(snap)
        ms.append(sc.step_profiled(DT)["fluid.pbf.neighbor_query"][0])
    snap.close()
    sc.close()
    print(pattern, ms)
    assert min(ms) < 9.0, ms
