"""A snapshot restored after the event stream was switched on or off: the
velocities, which worlds without springs keep in another form while nothing
reads them during a step, are those of the snapshot, and the steps and events
that follow are those of a world that had the stream in that state all along."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def spheres(n, springs=0.0):
    s = scenes.random_world(np.random.Generator(np.random.PCG64(n)), n, 0.05, 0.15, 0.5, 0.7, spring_frac=springs)
    s.dt = 1.0 / 120.0
    return s


WORLDS = {
    "resident": lambda: spheres(700),
    "spheres": lambda: spheres(5000),
    "springs": lambda: spheres(900, 0.2),
    "batch": lambda: scenes.pack([spheres(300 + k) for k in range(9)]),
    "jointed": lambda: scenes.jointed_bodies(seed=4, n=900, n_joints=200, n_springs=200, side=45.0),
}
CAP = 1 << 18


def state(w):
    b = w.read_bodies()
    return [b[k] for k in ("pos", "pos_old", "vel", "rotation", "angvel")]


def go_on(w, s, events):
    out = []
    for _ in range(2):
        w.step(s.dt)
        out.append(state(w) + (list(w.drain_events()) if events else []))
    return out


@pytest.mark.parametrize("steps", [0, 1, 2])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("events", [False, True])  # at the restore; the other at the snapshot
@pytest.mark.parametrize("name", list(WORLDS))
def test_restore_across_a_change_of_the_event_stream(name, events, pairs, steps):
    s = WORLDS[name]()

    def start(w, on):
        w.set_events(on, CAP)
        for _ in range(steps):
            w.step(s.dt)
        if pairs:
            w.emit_pairs(contacts_only=True)  # moves the storage, and V to its other buffer
        if on:
            w.drain_events()

    with native.World(s) as w:
        start(w, events)
        want = [state(w)] + go_on(w, s, events)
    with native.World(s) as w:
        start(w, not events)
        w.snapshot()
        w.rollout(s.dt, 3)
        w.set_events(events, CAP)
        for _ in range(2):
            w.restore()
            got = [state(w)] + go_on(w, s, events)
            for x, y in zip(got, want):
                assert len(x) == len(y)
                for a, b in zip(x, y):
                    assert np.array_equal(a, b)
