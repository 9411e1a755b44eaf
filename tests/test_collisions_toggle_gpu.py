"""Collisions switched off and on again between steps: the cells are counted
from zero when they come back, whatever the last substep with collisions left
in the counts -- a world that was switched steps on as a fresh world loaded
with its state does, bit for bit, on the resident, multi-kernel and general
paths, through steps, rollouts, pair emission and a restored snapshot."""
import copy

import numpy as np
import pytest

from blobs_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def spheres(n, springs=0.0):
    s = scenes.random_world(np.random.Generator(np.random.PCG64(n)), n, 0.05, 0.15, 0.5, 0.7, spring_frac=springs if n > 5 else 0.0)
    s.dt = 1.0 / 120.0
    return s


WORLDS = {
    "resident": lambda: spheres(700),
    "resident batch": lambda: scenes.pack([spheres(n, 0.1) for n in (300, 40, 900, 1, 64)]),
    "spheres": lambda: spheres(5000),
    "batch": lambda: scenes.pack([spheres(300 + k, 0.1) for k in range(20)] + [spheres(2600, 0.1)]),
    "jointed": lambda: scenes.jointed_bodies(seed=4, n=1500, n_joints=400, n_springs=500, side=55.0),
}


def collisions(w, on):
    w.cfg.collisions_enabled = 1 if on else 0
    native.check(native.lib().blobs_world_set_config(w._h, native.ctypes.byref(w.cfg)), "set_config")


def state(w):
    b = w.read_bodies()
    return [b[k] for k in ("pos", "pos_old", "vel", "rotation", "angvel")] + [w.read_snapshots()]


def fresh(w, s):
    """A world loaded with w's state."""
    f = copy.copy(s)
    f.pos, f.pos_old, f.vel, f.rotation, f.angvel, f.col_snap = state(w)
    f.vreq_set = np.zeros(s.n_bodies, np.uint8)
    return native.World(f, old_dt=float(np.float32(s.dt) / np.float32(s.substeps)))


@pytest.mark.parametrize("between", ["step", "rollout", "pairs", "restore"])
@pytest.mark.parametrize("name", list(WORLDS))
def test_counts_start_from_zero(name, between):
    s = WORLDS[name]()
    with native.World(s) as w:
        for _ in range(2):
            w.rollout(s.dt, 2)
            collisions(w, False)
            if between == "rollout":
                w.rollout(s.dt, 3)
            else:
                w.step(s.dt)
            if between == "pairs":
                w.emit_pairs(contacts_only=True)
            if between == "restore":
                w.snapshot()
            collisions(w, True)
            if between == "restore":
                w.step(s.dt)
                w.restore()
            with fresh(w, s) as f:
                before = w.contact_count()[0]
                for _ in range(2):
                    w.step(s.dt)
                    f.step(s.dt)
                    for a, b in zip(state(w), state(f)):
                        assert np.array_equal(a, b)
                assert w.contact_count()[0] - before == f.contact_count()[0]
