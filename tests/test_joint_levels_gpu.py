"""The small joint components' solves run level by level (k_joint_blocks)
against the oracle's sweep: chains of the longest kept component (64 joints,
256 levels over four iterations), stars, parallel joints, static ends, and
every number of iterations around the four that are laid out in levels.
Bodies of one collider: positions bit for bit; rotations as the joint path
states (CUDA's atan2f against the C library's)."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def chains(sizes, rng, star=False, doubled=False):
    """Components of the given joint counts, bodies in shuffled arena order."""
    n = sum(k + 1 for k in sizes)
    perm = rng.permutation(n)
    pos = np.zeros((n, 2), np.float32)
    a, b, at = [], [], 0
    for c, k in enumerate(sizes):
        ids = perm[at:at + k + 1]
        pos[ids] = np.stack([np.arange(k + 1) * 1.5, np.full(k + 1, 7.0 * c)], 1) + rng.uniform(-0.3, 0.3, (k + 1, 2))
        for i in range(k):
            a.append(ids[0] if star else ids[i])
            b.append(ids[i + 1])
        at += k + 1
    order = rng.permutation(len(a))  # arena order of the joints: any
    a, b = np.array(a)[order], np.array(b)[order]
    if doubled:
        a, b = np.concatenate([a, b[:len(b) // 2]]), np.concatenate([b, a[:len(a) // 2]])
    return pos, a, b


def world(sizes, iterations, seed, static=0.0, **kw):
    # radius 0.45: 1 / m_a + 1 / m_b = 1.1, below the 2 from which the reference's sweep diverges at a static end
    rng = np.random.Generator(np.random.PCG64(seed))
    pos, a, b = chains(sizes, rng, **kw)
    bt = (rng.random(len(pos)) < static).astype(np.uint8)
    s = scenes.spheres(pos, np.full(len(pos), 0.45, np.float32), rng.normal(0.0, 1.0, pos.shape).astype(np.float32),
                       body_type=bt)
    k = len(a)
    scenes.add_fixed_joints(s, a, b, rng.uniform(-0.2, 0.2, (k, 2)), rng.uniform(-0.2, 0.2, (k, 2)))
    s.jnt_distance *= np.float32(1.01)
    s.joint_iterations = iterations
    s.dt = 1.0 / 120.0
    return s


@pytest.mark.parametrize("iterations", [0, 1, 3, 4, 5, 9])
@pytest.mark.parametrize("sizes,kw", [([64], {}), ([1] * 300, {}), ([64, 63, 18, 9, 1] * 12, {"static": 0.1}),
                                      ([60, 30], {"star": True}), ([31, 20, 8], {"doubled": True}), ([70, 5], {})])
def test_sweeps_match_the_oracle(sizes, kw, iterations):
    s = world(sizes, iterations, seed=len(sizes) + iterations, **kw)
    with native.World(s) as w:
        order, colours = w.joint_order()
        w.step(s.dt)
        w.rollout(s.dt, 2)
        got = w.read_bodies()
    o = oracle.OracleWorld(s, 32, joint_order=order) if colours else oracle.OracleWorld(s, 32)
    assert o.step(s.dt, 3) == 0
    want = o.bodies()
    assert np.array_equal(got["pos"], want["pos"].astype(np.float32))
    assert np.array_equal(got["vel"], want["vel"].astype(np.float32))
    assert np.abs(got["rotation"] - want["rotation"]).max() <= 1e-5


@pytest.mark.parametrize("iterations", [2, 6])
def test_iterations_changed_after_loading(iterations):
    got = []
    for loaded in (4, iterations):
        s = world([64, 12, 3] * 5, loaded, seed=3)
        with native.World(s) as w:
            w.cfg.joint_iterations = iterations
            assert native.lib().blobs_world_set_config(w._h, w.cfg) == 0
            w.step(s.dt)
            got.append(w.read_bodies())
    assert np.array_equal(got[0]["pos"], got[1]["pos"]) and np.array_equal(got[0]["rotation"], got[1]["rotation"])
