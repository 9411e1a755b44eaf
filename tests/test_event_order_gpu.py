"""The event stream put in order on the device (events.cu) against the
oracle's list: batches that the device sorts (from 512 events), in one range
of (substep, collider) buckets and in several, bodies with many lower-id
contacts in one substep, and batches left over between drains."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def want_events(scene, steps):
    o = oracle.OracleWorld(scene, 32, record_events=True, grid_pairs=True)
    assert o.step(scene.dt, steps) == 0
    a, b, va, vb = o.events()
    return a, b, va.astype(np.float32), vb.astype(np.float32)


def same(got, want):
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


# 511 / 512 events stay below / reach the device; 40,000 colliders over 112
# substeps need two ranges of 2^22 buckets
@pytest.mark.parametrize("n,packing,steps", [(300, 0.3, 1), (3001, 0.5, 1), (20_011, 0.7, 2), (40_000, 0.4, 14)])
def test_sorted_batches(n, packing, steps):
    s = scenes.dense_spheres(seed=n, n=n, packing=packing)
    want = want_events(s, steps)
    with native.World(s) as w:
        w.set_events(True, 1 << 23)
        for _ in range(steps):
            w.step(s.dt)
        same(w.drain_events(), want)
        assert len(w.drain_events()[0]) == 0


def test_one_collider_touching_many():
    # the last body covers hundreds of lower ids: one bucket holds them all
    rng = np.random.Generator(np.random.PCG64(5))
    pos = rng.uniform(-2.0, 2.0, (900, 2)).astype(np.float32)
    pos[-1] = (0.01, 0.02)
    rad = np.full(900, 0.02, np.float32)
    rad[-1] = 2.0
    s = scenes.spheres(pos, rad, box=(-3.0, -3.0, 3.0, 3.0))
    # one substep: the next ones pile spheres up in the corners, where coincident centres take the push-out branch
    s.dt, s.substeps = 1.0 / 240.0, 1
    o = oracle.OracleWorld(s, 32, record_events=True)
    assert o.step(s.dt, 1) == 0
    a, b, va, vb = o.events()
    with native.World(s) as w:
        w.set_events(True, 1 << 20)
        w.step(s.dt)
        got = w.drain_events()
    assert len(got[0]) > 512
    same(got, (a, b, va.astype(np.float32), vb.astype(np.float32)))


def test_left_over_batches_keep_their_order():
    s = scenes.dense_spheres(seed=77, n=5000, packing=0.6)
    want = want_events(s, 3)
    got = []
    with native.World(s) as w:
        w.set_events(True, 1 << 22)
        w.step(s.dt)
        got.append(w.drain_events(cap=700))      # part of a device batch
        w.step(s.dt)
        got.append(w.drain_events(cap=100))      # the rest of it moves ahead of the second batch
        got.append(w.drain_events(cap=0))
        w.step(s.dt)
        got.append(w.drain_events())
    same([np.concatenate([g[k] for g in got]) for k in range(4)], want)
