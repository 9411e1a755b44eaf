"""Event batches of exactly the count from which the device sorts them (512 in
one range of buckets), one less and one more, against the oracle's order."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("events", [1, 511, 512, 513])
def test_batches_around_the_device_sort(events):
    rng = np.random.Generator(np.random.PCG64(events))
    at = np.stack([np.arange(events) % 32, np.arange(events) // 32], 1).astype(np.float32) * np.float32(3.0)
    pos = np.concatenate([at, at + np.float32((0.15, 0.05))])[rng.permutation(2 * events)]
    s = scenes.spheres(pos, np.full(2 * events, 0.1, np.float32), rng.normal(0.0, 0.1, pos.shape).astype(np.float32))
    s.dt, s.substeps = 1.0 / 240.0, 1
    o = oracle.OracleWorld(s, 32, record_events=True)
    assert o.step(s.dt, 1) == 0
    want = o.events()
    assert len(want[0]) == events
    with native.World(s) as w:
        w.set_events(True, 1 << 12)
        w.step(s.dt)
        got = w.drain_events()
    for g, x in zip(got, want):
        assert np.array_equal(g, x.astype(g.dtype))
