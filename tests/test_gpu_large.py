"""Parity of large single scenes (at least 2^18 particles), where the
constraint, XSPH and vorticity passes take the warp-cooperative neighbour
walk: the exact build must still equal the oracle bit for bit.

The cases cover warps that sit in one cell (a lattice whose cells hold 4 x 4 x 4
particles), warps that straddle two or three cells of a row (h = 3.5 r, so
cells hold 27 to 64 particles), the second step of the configured dam break
(the first one scatters the lattice, so warps straddle rows and cells fill
unevenly), the plain 27-cell neighbourhood (hash_compat 0) and the reference's
hash buckets near the axes (a block at the origin).
"""
import numpy as np
import pytest

from novaphy_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def run_both(port_mt, w, nsteps, **kw):
    from oracle.oracle import Settings

    st = dict(w.settings)
    st.update(kw)
    sc = capi.Scene(capi.default_settings(**st, exact_arithmetic=1), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    sc.step(w.dt, nsteps)
    got = sc.state()
    sc.close()
    ost = {k: v for k, v in st.items() if k not in ("exact_arithmetic", "hash_compat")}
    z = np.zeros(w.n, np.float32)
    want = port_mt.steps(Settings.make(**ost), w.x, w.v, z, z, w.dt, w.gravity, w.mass, nsteps)
    return got, want


def assert_equal(got, want, tag):
    for name, a, b in zip("x v rho lam".split(), got, want):
        bad = np.flatnonzero(~((a == b) | (np.isnan(a) & np.isnan(b))).reshape(len(a), -1).all(1))
        assert bad.size == 0, (tag, name, bad[:5], bad.size)


@pytest.mark.parametrize("nsteps", [1, 2])
def test_lattice_block_one_cell_per_warp(port_mt, nsteps):
    w = workloads.dam_break((64, 64, 64), 0.01, (4.0, 2.0, 2.0), dt=1.0 / 240.0, jitter=1e-5,
                            seed=5, vorticity=1e-4)
    assert w.n >= 1 << 18
    assert_equal(*run_both(port_mt, w, nsteps), ("lattice", nsteps))


def test_warps_straddle_cells(port_mt):
    # h = 3.5 r: cells of 27 to 64 particles, so warps span two or three
    # cells of a row, or two rows.
    w = workloads.dam_break((66, 64, 64), 0.01, (4.0, 2.0, 2.0), h_factor=3.5, dt=1.0 / 240.0,
                            jitter=1e-5, seed=6, vorticity=1e-4)
    assert w.n >= 1 << 18
    assert_equal(*run_both(port_mt, w, 2), "straddle")


@pytest.mark.parametrize("kw", [dict(hash_compat=0), dict(vorticity_epsilon=0.0),
                                dict(corr_k=0.001, corr_delta_q=0.3, xsph_viscosity=0.0)])
def test_large_settings_variants(port_mt, kw):
    w = workloads.dam_break((64, 64, 65), 0.01, (4.0, 2.0, 2.0), dt=1.0 / 240.0, jitter=1e-5,
                            seed=7, vorticity=1e-4)
    nsteps = 2
    if kw.get("hash_compat") == 0:
        # Away from the axes the reference's buckets are the plain 27 cells.
        # One step only: the configured s_corr scatters the block over the
        # whole box in the first step, and particles that reach the walls at
        # the axes fall into merged buckets in the second.
        shift = np.array([0.5, 0.25, 0.25], np.float32)
        w.x = (w.x + shift).astype(np.float32)
        xp = port_mt.predict(w.x, w.v, w.dt, w.gravity)[0]
        assert port_mt.hash_collisions(xp, np.float32(w.settings["kernel_radius"])) == 0
        nsteps = 1
    assert_equal(*run_both(port_mt, w, nsteps, **kw), kw)


@pytest.mark.parametrize("exact", [1, 0])
def test_density_first_walk_equals_single_walk(port_mt, exact):
    """The density pass of a large scene may sum the densities alone first and
    then walk again for the gradients of the lanes with C_i >= 0, in the
    iterations where few warps needed gradients in the scene's previous step;
    a scene's first step has no such record and walks once.  Stepping the
    same state again (after the configured first step, iterations 1-3 have
    almost no C_i >= 0) must give the same bits, and in the exact build the
    oracle's."""
    w = workloads.dam_break((64, 64, 64), 0.01, (4.0, 2.0, 2.0), dt=1.0 / 240.0, jitter=1e-5,
                            seed=5, vorticity=1e-4)
    sc = capi.Scene(capi.default_settings(**w.settings, exact_arithmetic=exact), w.x, w.v,
                    mass=w.mass)
    sc.set_gravity(w.gravity)
    snap = sc.snapshot()
    runs = []
    for _ in range(3):
        sc.restore(snap)
        sc.step(w.dt)
        runs.append(sc.state())
    sc.close()
    for r in runs[1:]:
        assert_equal(r, runs[0], ("again", exact))
    if exact:
        from oracle.oracle import Settings

        z = np.zeros(w.n, np.float32)
        want = port_mt.steps(Settings.make(**w.settings), w.x, w.v, z, z, w.dt, w.gravity,
                             w.mass, 1)
        assert_equal(runs[2], want, "oracle")


def clump_block(nclump, seed=9):
    """The 64^3 lattice with nclump extra particles at one point, bit for bit
    (x, v = 0), inside the block in cell (5, 5, 5): half of them inserted in
    the index order between the lattice's z-layers 21 and 22 (so members of
    that cell sit between the two halves in cell order) and half at the end."""
    w = workloads.dam_break((64, 64, 64), 0.01, (4.0, 2.0, 2.0), dt=1.0 / 240.0, jitter=1e-5,
                            seed=seed, vorticity=1e-4)
    p = np.full((nclump, 3), 0.205, np.float32)
    half = nclump // 2
    cut = 64 * 64 * 22
    w.x = np.concatenate([w.x[:cut], p[:half], w.x[cut:], p[half:]]).astype(np.float32)
    w.v = np.zeros_like(w.x)
    return w


@pytest.mark.parametrize("nsteps", [1, 2])
def test_runs_of_identical_particles(port_mt, nsteps):
    """Particles with bit-identical state next to each other in cell order
    (runs) come out identical: the run's first particle computes and writes
    its results for the others, and as candidates the run's particles add
    their term in one exact repeated addition (cell ranges and rows of at
    least 1,024 candidates).  Two runs of 1,500 in one cell, with members of
    the lattice between them: the oracle's bits after one and two steps."""
    w = clump_block(3000)
    assert w.n >= 1 << 18
    assert_equal(*run_both(port_mt, w, nsteps), ("runs", nsteps))


def test_runs_with_default_scorr(port_mt):
    """The same with PBFSettings' own s_corr."""
    w = clump_block(2400, seed=10)
    got, want = run_both(port_mt, w, 2, corr_k=0.001, corr_delta_q=0.3)
    assert_equal(got, want, "runs default s_corr")


def pile_block(n, lengths, seed, same):
    """A lattice of 2^18 and more particles and, in one cell of the upper half of its box, n particles: runs of
    bit-identical ones of the given lengths in turn (same), or all different, in random places of the order."""
    w = workloads.dam_break((64, 64, 64), 0.02, (3.0, 3.0, 3.0), jitter=1e-4, seed=seed, vorticity=1e-4)
    rng = np.random.default_rng(seed)
    h = w.settings["kernel_radius"]
    at = (2.0 + h * 0.3 + 0.3 * h * rng.random((n, 3))).astype(np.float32)
    if same:
        k = 0
        while k < n:
            m = min(int(lengths[rng.integers(len(lengths))]), n - k)
            at[k:k + m] = at[k]
            k += m
    w.x = np.concatenate([w.x, at]).astype(np.float32)
    w.v = np.zeros_like(w.x)
    return w


@pytest.mark.parametrize("lengths", [(1, 2, 3, 5), (1, 31, 33, 63, 64, 65, 97, 200)])
def test_runs_of_every_length(port_mt, lengths):
    """Runs too short to be taken as one candidate between longer ones and single particles, in a cell of more
    candidates than a list holds: the oracle's bits after one and two steps."""
    for nsteps in (1, 2):
        w = pile_block(5000, lengths, 21, True)
        assert_equal(*run_both(port_mt, w, nsteps), ("lengths", lengths, nsteps))


def test_a_pile_of_short_runs_costs_no_more_than_one_of_different_particles():
    """A cell of 20,000 particles, many of them bit-identical in twos to eights, against the same cell with
    all particles different: the identical ones save work and may not cost any (they cost 2.5 times as much when each
    run was taken as a candidate of its own)."""
    ms = []
    for same in (True, False):
        w = pile_block(20000, (1, 2, 2, 3, 5, 8), 23, same)
        sc = capi.Scene(capi.default_settings(**w.settings), w.x, w.v, mass=w.mass)
        sc.set_gravity(w.gravity)
        seed = sc.snapshot()
        sc.replay_timed(seed, w.dt, 1)
        ms.append(min(sc.replay_timed(seed, w.dt, 1) for _ in range(3)))
        seed.close()
        sc.close()
    assert ms[0] < 1.2 * ms[1], ms
