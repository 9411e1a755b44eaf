"""A snapshot holds what later steps read and no more: after steps of another
length, host writes, pair emission and event toggling have gone over
everything else, a restored world steps as the one that was never disturbed
-- taken from either storage buffer, with V in the other one, before and
after the first step, on the resident, multi-kernel and general paths."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def spheres(n, springs=0.0):
    s = scenes.random_world(np.random.Generator(np.random.PCG64(n)), n, 0.05, 0.15, 0.5, 0.7, spring_frac=springs)
    s.dt = 1.0 / 120.0
    return s


def turning():
    s = spheres(2500)
    s.angvel = np.linspace(-1.0, 1.0, 2500, dtype=np.float32)
    s.body_type[::17] = 1
    return s


WORLDS = {
    "resident": lambda: spheres(700),
    "resident springs": lambda: spheres(700, 0.3),
    "spheres": lambda: spheres(5000),
    "springs": lambda: spheres(5000, 0.2),
    "turning": turning,
    "batch": lambda: scenes.pack([spheres(300 + k, 0.1) for k in range(40)] + [spheres(2600, 0.1)]),
    "jointed": lambda: scenes.jointed_bodies(seed=4, n=1500, n_joints=400, n_springs=500, side=55.0),
}


def state(w):
    return [w.read_bodies()[k] for k in ("pos", "pos_old", "vel", "rotation", "angvel")] + [
        w.read_snapshots(), np.array(w.contact_count())]


@pytest.mark.parametrize("steps", [0, 1, 2])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("name", list(WORLDS))
def test_restored_world_goes_on_undisturbed(name, steps, pairs):
    s = WORLDS[name]()

    def start(w):
        for _ in range(steps):
            w.step(s.dt)
        if pairs:
            w.emit_pairs(contacts_only=True)  # moves the storage, and V to its other buffer

    def go_on(w):
        out = [state(w)]
        w.step(s.dt)
        out.append(state(w))
        w.rollout(s.dt, 3)
        return out + [state(w)]

    with native.World(s) as w:
        start(w)
        want = go_on(w)
    with native.World(s) as w:
        start(w)
        w.snapshot()
        for again in range(2):
            w.rollout(s.dt * 0.7, 2 + again)
            w.emit_pairs(contacts_only=False)
            w.write_bodies(pos=np.ascontiguousarray(s.pos[::-1]), vel=np.ones_like(s.pos))
            w.set_events(True, 1 << 20)
            w.step(s.dt)
            w.set_events(False)
            w.restore()
            for a, b in zip(go_on(w), want):
                for x, y in zip(a, b):
                    assert np.array_equal(x, y)
