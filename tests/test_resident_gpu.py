"""Whole steps of small worlds in one launch (k_resident) against the kernels
of a substep, which run while phase timing is on: states, contacts, deferred
bodies and what later calls make of the state, bit for bit -- over the edges
of its blocks (256 bodies), clusters and rule, over uniform worlds and worlds
with per-body records, and over odd numbers of substeps and steps (cell
counts, keys and ranks end up in another buffer)."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def state(w):
    return w.read_bodies(), w.read_snapshots(), w.contact_count(), w.pushout_count(), w.deferred_count()


def same(x, y):
    for k in x[0]:
        assert np.array_equal(x[0][k], y[0][k], equal_nan=True), k
    assert np.array_equal(x[1], y[1]) and x[2:] == y[2:]


def both(scene, drive):
    got = []
    for phases in (False, True):
        with native.World(scene) as w:
            w.set_timing(phases)
            before = w.kernel_launches()
            got.append((drive(w), w.kernel_launches() - before))
    return got


def check(scene, steps=3, resident=True):
    def drive(w):
        out = []
        w.step(scene.dt)            # velocity requests pending, dt / old_dt
        out.append(state(w))
        w.rollout(scene.dt, steps)  # one graph
        out.append(state(w))
        pairs = w.emit_pairs(contacts_only=True)
        w.step(scene.dt * 0.5)      # another dt, after a call that took the cell counts
        out.append(state(w))
        return out, pairs
    (a, ka), (b, kb) = both(scene, drive)
    for x, y in zip(a[0], b[0]):
        same(x, y)
    assert np.array_equal(a[1], b[1])
    assert (ka < kb) == resident


def single(n, packing, seed=0, springs=0.0, statics=0.0):
    rng = np.random.Generator(np.random.PCG64(1000 * n + seed))
    s = scenes.random_world(rng, n, 0.05, 0.15, packing, 0.7, spring_frac=springs if n > 5 else 0.0)
    if statics:
        s.body_type = (rng.random(n) < statics).astype(np.uint8)
    s.dt = 1.0 / 120.0
    return s


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 511, 513, 1024, 1025, 2047, 2048, 2049])
def test_block_and_cluster_edges(n):
    check(single(n, 0.5), resident=n <= 2048)


@pytest.mark.parametrize("n,packing,springs,statics", [(700, 0.3, 0.1, 0.0), (700, 0.3, 0.6, 0.0), (900, 0.5, 0.2, 0.05),
                                                       (300, 2.5, 0.0, 0.0), (2000, 3.0, 0.3, 0.02)])
def test_springs_static_bodies_and_crowds(n, packing, springs, statics):
    # packing 2.5 and 3: bodies with more candidates or near candidates than the kernels take in line
    check(single(n, packing, springs=springs, statics=statics))


@pytest.mark.parametrize("substeps,steps", [(1, 1), (1, 4), (3, 5), (7, 2), (8, 130), (1100, 1)])
def test_odd_substeps_and_long_rollouts(substeps, steps):
    s = single(400, 0.6)
    s.substeps = substeps
    check(s, steps=steps)


def test_circles_rotation_and_gravity_scales():
    s = single(500, 0.4)
    rng = np.random.Generator(np.random.PCG64(9))
    s.circles = np.array([[0.0, 0.0, 3.0]], np.float32)
    s.angvel = rng.normal(0.0, 1.0, 500).astype(np.float32)
    s.gravity_mod = rng.uniform(0.0, 2.0, 500).astype(np.float32)
    check(s)


@pytest.mark.parametrize("counts,springs", [([1, 2, 300, 1500, 2048, 64], 0.1), ([513] * 16, 0.5),
                                            ([64 + 7 * k for k in range(64)], 0.0), ([40] * 300, 0.2),
                                            ([700, 5, 900, 256] * 35, 0.0)])
@pytest.mark.parametrize("statics", [0.0, 0.05])
def test_batches(counts, springs, statics):
    s = scenes.pack([single(n, 0.35, seed=k, springs=springs, statics=statics) for k, n in enumerate(counts)])
    s.dt = 1.0 / 120.0
    check(s, steps=2)


def test_writes_snapshots_and_streams():
    import torch
    s = single(1500, 0.5)

    def drive(w):
        out = []
        w.step(s.dt)
        w.snapshot()
        w.rollout(s.dt, 3)
        first = state(w)
        w.restore()
        stream = torch.cuda.Stream()
        w.set_stream(stream.cuda_stream)
        w.rollout(s.dt, 3)
        same(state(w), first)
        w.set_stream(0)
        pos = np.ascontiguousarray(s.pos[::-1])
        w.write_bodies(pos=pos, vel=np.ones_like(pos))
        w.rollout(s.dt, 2)
        out.append(state(w))
        w.set_events(True, 1 << 20)   # the kernels of a substep from here on
        w.step(s.dt)
        out.append(w.drain_events())
        w.set_events(False)
        w.step(s.dt)
        return out + [state(w)]
    (a, _), (b, _) = both(s, drive)
    same(a[0], b[0])
    same(a[2], b[2])
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)
