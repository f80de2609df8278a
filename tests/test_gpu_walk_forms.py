"""The forms of the neighbour walk (teams of 8 and 16 particles, warps of 32) against the oracle, bit for
bit: particle counts at the edges of each form's range and of its tiles, and the states that each path of the
walk takes: cells of 8 to 64 particles (warps and teams that straddle cells), merged reference buckets (a block
at the origin), the plain 27-cell neighbourhood, particles thrown far apart (groups too wide for the fp16
distance test, teams over many cells), candidates piled into one cell (more terms than a list holds), and a
support radius outside the range of the paired arithmetic."""
import numpy as np
import pytest

from novaphy_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def block(n, h_factor=4.0, seed=0, r=0.02, **kw):
    """The first n particles of a jittered lattice with velocities, in a box twice its size."""
    e = int(np.ceil(n ** (1.0 / 3.0)))
    w = workloads.dam_break((e, e, e), r, (2.0 * e * r + r,) * 3, h_factor=h_factor, jitter=0.05 * r, seed=seed,
                            **kw)
    rng = np.random.default_rng(seed + 1)
    w.x = w.x[:n].copy()
    w.v = (rng.normal(size=w.x.shape) * 0.2).astype(np.float32)
    return w


def check(port_mt, w, nsteps=1, **kw):
    from oracle.oracle import Settings

    st = dict(w.settings, **kw)
    sc = capi.Scene(capi.default_settings(**st, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.step(w.dt, nsteps)
    got = sc.state()
    sc.close()
    ost = {k: v for k, v in st.items() if k != "hash_compat"}
    z = np.zeros(w.n, np.float32)
    want = port_mt.steps(Settings.make(**ost), w.x, w.v, z, z, w.dt, w.gravity, w.mass, nsteps)
    for name, a, b in zip("x v rho lam".split(), got, want):
        bad = np.flatnonzero(~((a == b) | (np.isnan(a) & np.isnan(b))).reshape(len(a), -1).all(1))
        assert bad.size == 0, (name, bad[:5], bad.size)


# One particle, part of a tile, whole tiles and one more, and both sides of the lines between the forms.
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 1000, 8191, 8192, 8209, 131071, 131072, 131105])
def test_sizes(port_mt, n):
    check(port_mt, block(n, vorticity=1e-4 if n % 2 else 0.0))


@pytest.mark.parametrize("n", [3000, 40000, 140000])
@pytest.mark.parametrize("h_factor", [2.0, 2.9, 3.5])
def test_cells_of_few_particles(port_mt, n, h_factor):
    check(port_mt, block(n, h_factor=h_factor, seed=3, vorticity=1e-4), 2, corr_k=0.001, corr_delta_q=0.3)


@pytest.mark.parametrize("n", [3000, 40000, 140000])
def test_far_and_scattered(port_mt, n):
    # One in 20 particles leaves with up to 40 h a step; without walls most of them alias into the grid.
    w = block(n, seed=5, vorticity=1e-4)
    rng = np.random.default_rng(7)
    far = rng.random(n) < 0.05
    w.v[far] *= np.float32(40.0 * w.settings["kernel_radius"] / w.dt)
    check(port_mt, w, 2)
    check(port_mt, w, 1, use_domain_bounds=0)


@pytest.mark.parametrize("n", [3000, 40000, 140000])
def test_more_terms_than_a_list_holds(port_mt, n):
    w = block(n, seed=9, vorticity=1e-4)
    rng = np.random.default_rng(11)
    pile = rng.permutation(n)[: 1400]
    w.x[pile] = (0.13 + 0.01 * rng.random((1400, 3))).astype(np.float32)
    w.v[pile] = 0.0
    check(port_mt, w, 1)


@pytest.mark.parametrize("n", [3000, 40000, 140000])
@pytest.mark.parametrize("scale", [0.005, 2000.0])
def test_radius_outside_the_paired_range(port_mt, n, scale):
    w = block(n, seed=13, r=0.02 * scale, vorticity=1e-4)
    check(port_mt, w, 1)


@pytest.mark.parametrize("n", [3000, 40000, 140000])
def test_plain_neighbourhood_away_from_the_axes(port_mt, n):
    # Far from the axes no two cells of a neighbourhood share a reference key, so hash_compat 0 is the
    # reference's step too.
    w = block(n, seed=15)
    shift = np.float32(7.0)
    w.x = (w.x + shift).astype(np.float32)
    lo, hi = (7.0,) * 3, tuple(7.0 + t for t in w.settings["domain_upper"])
    check(port_mt, w, 1, domain_lower=lo, domain_upper=hi, hash_compat=0)


@pytest.mark.parametrize("n", [1, 700, 9000, 140000])
def test_merged_buckets(port_mt, n):
    # A block around the origin, where cells on both sides of the axes share reference keys; the scene held
    # more particles before, and some leave the grid, so that runs of cells alternate within slots.
    from oracle.oracle import Settings

    big, w = block(n + 5000, seed=19), block(n, seed=17, vorticity=1e-4)
    w.x = (w.x - w.x.mean(0)).astype(np.float32)
    out = np.random.default_rng(21).random(n) < 0.03
    w.v[out] *= np.float32(15.0 * w.settings["kernel_radius"] / w.dt)
    half = tuple(0.75 * t for t in w.settings["domain_upper"])
    st = dict(w.settings, domain_lower=tuple(-t for t in half), domain_upper=half)
    sc = capi.Scene(capi.default_settings(**st, exact_arithmetic=1), big.x, big.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.step(w.dt, 1)
    sc.reset(w.x, w.v)
    sc.step(w.dt, 2)
    got = sc.state()
    sc.close()
    z = np.zeros(w.n, np.float32)
    want = port_mt.steps(Settings.make(**st), w.x, w.v, z, z, w.dt, w.gravity, w.mass, 2)
    for name, a, b in zip("x v rho lam".split(), got, want):
        assert np.array_equal(a, b), name
