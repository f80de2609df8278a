"""The memory of kept lists: any other allocation of the library that finds no room gets it, it goes back to the
device with its scene, a refusal does not last, and steps with and without lists leave the same bits, in scenes and
batches on both sides of the line between teams and warps."""
import gc

import numpy as np
import pytest

from novaphy_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

GB = 1 << 30


def lattice(e, r=0.02, seed=1, h_factor=2.0, **kw):
    w = workloads.dam_break((e, e, e), r, (2.0 * e * r,) * 3, h_factor=h_factor, jitter=0.05 * r, seed=seed, **kw)
    rng = np.random.default_rng(seed)
    w.v = (0.2 * rng.normal(size=w.x.shape)).astype(np.float32)
    return w


def scene(w, **kw):
    sc = capi.Scene(capi.default_settings(**w.settings, **kw), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)
    return sc


def state(sc):
    sc.sync()
    return [a.view(np.uint32) for a in sc.state()]


def list_bytes(n):
    return 2 * 1024 * n  # 256 rows of two positions


def free_bytes():
    import torch

    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def ballast():
    """ballast.take(leave) takes all but `leave` bytes of the device, ballast.free() gives them back."""
    import torch

    class Ballast:
        held = None

        def take(self, leave):
            self.held = torch.empty(max(free_bytes() - leave, 0), dtype=torch.uint8, device="cuda")

        def free(self):
            self.held = None
            free_bytes()

    b = Ballast()
    yield b
    b.free()


def test_a_closed_scene_gives_its_lists_back():
    w = lattice(160)  # 4,096,000 particles: 8.4 GB of lists
    before = free_bytes()
    sc = scene(w)
    sc.step(w.dt)
    assert capi.scene_device_bytes(sc) > list_bytes(w.n)
    rest = capi.scene_device_bytes(sc) - list_bytes(w.n)
    sc.close()
    assert before - free_bytes() < rest + 4.5 * GB


def test_lists_give_way(ballast):
    w = lattice(160)
    a = scene(w)
    a.step(w.dt)
    with_lists = capi.scene_device_bytes(a)
    assert with_lists > list_bytes(w.n)
    big = lattice(200, seed=3)  # 8,000,000 particles: 3.3 GB without lists
    ballast.take(GB // 2)
    b = scene(big)
    b.step(big.dt)  # no room but that of a's lists
    assert capi.scene_device_bytes(a) < with_lists - list_bytes(w.n) // 2
    snap = b.snapshot()
    a.step(w.dt)
    got = state(a)
    for o in (snap, a, b):
        o.close()
    ballast.free()
    ref = scene(w)
    ref.set_kept_lists(False)
    ref.step(w.dt, 2)
    assert all(np.array_equal(x, y) for x, y in zip(got, state(ref)))
    ref.close()


def test_a_refusal_does_not_last(ballast):
    w = lattice(160)
    sc = scene(w)
    snap = sc.snapshot()
    ballast.take(5 * GB // 2)
    sc.step(w.dt)
    without = capi.scene_device_bytes(sc)
    assert without < list_bytes(w.n)
    ballast.free()
    for _ in range(80):
        sc.restore(snap)  # the same step each time, not a pile's
        sc.step(w.dt, sync=False)
    sc.sync()
    assert capi.scene_device_bytes(sc) > list_bytes(w.n)
    snap.close()
    sc.close()


@pytest.mark.parametrize("e", [15, 40, 52, 66])  # teams of 8, of 16, warps
@pytest.mark.parametrize("exact", [1])
def test_same_bits_without_lists(e, exact):
    w = lattice(e, h_factor=4.0, vorticity=1e-4)
    w.settings.update(corr_k=0.001, corr_delta_q=0.3)
    out = []
    for on in (True, False):
        sc = scene(w, exact_arithmetic=exact)
        sc.set_kept_lists(on)
        sc.step(w.dt, 2)
        assert (capi.scene_device_bytes(sc) > list_bytes(w.n)) == on
        sc.set_kept_lists(not on)
        sc.step(w.dt, 1)
        out.append(state(sc))
        sc.close()
    assert all(np.array_equal(x, y) for x, y in zip(*out))


@pytest.mark.parametrize("edges", [(9, 14, 11), (44, 30, 40)])  # teams, warps
def test_same_bits_without_lists_in_a_batch(edges):
    ws = [lattice(e, seed=e, h_factor=4.0, vorticity=1e-4 if k else 0.0, iterations=2 + k)
          for k, e in enumerate(edges)]
    out = []
    for on in (True, False):
        scs, b = [scene(w) for w in ws], capi.Batch()
        b.set_kept_lists(on)
        b.step(scs, [w.dt for w in ws], [2] * len(ws))
        assert (b.device_bytes() > list_bytes(sum(w.n for w in ws))) == on
        out.append([x for sc in scs for x in state(sc)])
        for o in scs + [b]:
            o.close()
    assert all(np.array_equal(x, y) for x, y in zip(*out))
