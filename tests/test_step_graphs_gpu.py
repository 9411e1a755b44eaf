"""Steps and rollouts used again and again: launched kernel by kernel the
first time from a storage buffer, captured into a graph the second, replayed
after that (a step of eight substeps moves the state to the other buffer, so
five uses reach every one of them from both).  The states after each use
against the oracle, and, where worlds are run in classes by their size --
forked and joined inside the graph -- against the kernels of a substep."""
import ctypes

import numpy as np
import pytest

from blobs_gb300 import native, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu

USES = 5


def spheres(n, packing=0.4, springs=0.0):
    s = scenes.random_world(np.random.Generator(np.random.PCG64(n)), n, 0.05, 0.15, packing, 0.7, spring_frac=springs)
    s.dt = 1.0 / 120.0
    return s


def exact(got, want):
    for k in ("pos", "pos_old", "vel"):
        assert np.array_equal(got[k].astype(np.float64), want[k]), k


@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("n,springs", [(500, 0.0), (2500, 0.0), (2500, 0.2), (30_000, 0.0)])
def test_repeated_rollouts_match_the_oracle(n, springs, steps):
    s = spheres(n, springs=springs)
    o = oracle.OracleWorld(s, 32, grid_pairs=True)
    with native.World(s) as w:
        w.step(s.dt)
        assert o.step(s.dt, 1) == 0
        for _ in range(USES):
            w.rollout(s.dt, steps)
            assert o.step(s.dt, steps) == 0
            exact(w.read_bodies(), o.bodies())
        assert w.contact_count()[0] == o.contacts


def test_repeated_rollouts_of_multi_collider_bodies():
    s = scenes.jointed_bodies(seed=4, n=1500, n_joints=0, n_springs=500, side=55.0)
    o = oracle.OracleWorld(s, 32, grid_pairs=True)
    with native.World(s) as w:
        w.step(s.dt)
        assert o.step(s.dt, 1) == 0
        for _ in range(USES):
            w.rollout(s.dt, 3)
            assert o.step(s.dt, 3) == 0
            exact(w.read_bodies(), o.bodies())


@pytest.mark.parametrize("joints", [0, 400])  # the springs on a branch of their own inside the graph
def test_repeated_rollouts_match_single_steps(joints):
    s = scenes.jointed_bodies(seed=5, n=1500, n_joints=joints, n_springs=500, side=55.0)
    with native.World(s) as w, native.World(s) as plain:
        plain.set_timing(True)  # no branches
        for f in (w, plain):
            f.step(s.dt)
        for _ in range(USES):
            w.rollout(s.dt, 3)
            for _ in range(3):
                plain.step(s.dt)
            a, b = w.read_bodies(), plain.read_bodies()
            for k in a:
                assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("rollout", [False, True])
@pytest.mark.parametrize("n", [400, 3000])
def test_events_of_repeated_rollouts(n, rollout):
    s = scenes.dense_spheres(seed=n, n=n, packing=0.4)
    o = oracle.OracleWorld(s, 32, record_events=True, grid_pairs=True)
    seen = 0
    with native.World(s) as w:
        w.set_events(True, 1 << 21)
        for _ in range(USES):
            if rollout:
                w.rollout(s.dt, 2)
            else:
                w.step(s.dt)
                w.step(s.dt)
            got = w.drain_events()
            assert o.step(s.dt, 2) == 0
            want = [x[seen:] for x in o.events()]
            seen += len(want[0])
            for g, x in zip(got, want):
                assert np.array_equal(g, x.astype(g.dtype))
    assert seen > 0


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("counts", [[40, 300, 900, 1500], [700, 5, 900, 256] * 20])
def test_repeated_rollouts_in_classes(counts, steps):
    s = scenes.pack([spheres(n, 0.35, 0.1 if n > 5 else 0.0) for n in counts])
    s.dt = 1.0 / 120.0
    with native.World(s) as w, native.World(s) as phases:
        phases.set_timing(True)
        launches = []
        for f in (w, phases):
            f.step(s.dt)
            launches.append(f.kernel_launches())
        for _ in range(USES):
            for f in (w, phases):
                f.rollout(s.dt, steps)
            a, b = w.read_bodies(), phases.read_bodies()
            for k in a:
                assert np.array_equal(a[k], b[k]), k
            assert np.array_equal(w.read_snapshots(), phases.read_snapshots())
            assert w.contact_count() == phases.contact_count()
        classes = w.kernel_launches() - launches[0]
        assert 2 * USES <= classes < (phases.kernel_launches() - launches[1]) / 4


def test_graphs_on_a_stream_of_the_callers():
    """Captured on the world's own stream, replayed on the caller's, and after
    that stream is destroyed on the world's again, checkpoints of a recorded
    rollout that were last used on it included."""
    import torch
    s = spheres(2500, springs=0.1)
    g = np.ones((s.n_bodies, 2), np.float32)
    rt = torch.cuda.cudart()
    with native.World(s) as w, native.World(s) as plain:
        for f in (w, plain):
            for _ in range(4):
                f.rollout(s.dt, 2)
        handle = ctypes.c_void_p()
        assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
        w.set_stream(handle.value)
        for f in (w, plain):
            for _ in range(2):
                f.rollout(s.dt, 2)
            f.rollout_record(s.dt, 4, 2)
        a, b = w.backward(g, s.n_springs), plain.backward(g, s.n_springs)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        w.set_stream(0)
        assert int(rt.cudaStreamDestroy(handle.value)) == 0
        for f in (w, plain):
            f.rollout_record(s.dt, 2, 1)  # frees the checkpoints used on that stream
            f.rollout(s.dt, 2)
        a, b = w.read_bodies(), plain.read_bodies()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
