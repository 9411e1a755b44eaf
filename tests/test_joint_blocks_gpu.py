"""Joint blocks by levels and in turn -- one or the other by the components and
the number of iterations, both in worlds whose blocks differ -- against the
oracle's sweep.  Bodies of one collider: positions bit for bit; rotations as the joint
path states (CUDA's atan2f against the C library's)."""
import numpy as np
import pytest

from blobs_gb300 import native
from oracle import oracle
from test_joint_levels_gpu import world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iterations", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("sizes,kw", [([64] * 3 + [1] * 700, {}), ([40, 2] + [3] * 500, {"star": True}),
                                      ([64, 20] * 2 + [2] * 600, {"doubled": True, "static": 0.05})])
def test_both_kinds_of_blocks_match_the_oracle(sizes, kw, iterations):
    s = world(sizes, iterations, seed=7 * len(sizes) + iterations, **kw)
    with native.World(s) as w:
        order, colours = w.joint_order()
        for _ in range(3):
            w.step(s.dt)
        got = w.read_bodies()
    o = oracle.OracleWorld(s, 32, joint_order=order) if colours else oracle.OracleWorld(s, 32)
    assert o.step(s.dt, 3) == 0
    want = o.bodies()
    assert np.array_equal(got["pos"], want["pos"].astype(np.float32))
    assert np.array_equal(got["vel"], want["vel"].astype(np.float32))
    assert np.abs(got["rotation"] - want["rotation"]).max() <= 1e-5
