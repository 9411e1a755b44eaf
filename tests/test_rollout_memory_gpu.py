"""Checkpoints and reverse-pass scratch come from a pool shared by every
world and stream: gradients do not depend on what used the memory before, on
whose stream it was used, or on that stream being gone."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def batch(seed, n):
    rng = np.random.Generator(np.random.PCG64(seed))
    return scenes.pack([scenes.random_world(rng, n + 7 * k, 0.1, 0.2, 0.3, 1.0, spring_frac=0.3) for k in range(3)])


def gradients(w, s, steps, every):
    w.restore()
    w.rollout_record(1.0 / 60.0, steps, every)
    g = np.linspace(-1.0, 1.0, 2 * s.n_bodies, dtype=np.float32).reshape(-1, 2)
    return w.backward(g, s.n_springs)


def test_gradients_with_reused_memory():
    import torch
    small, large = batch(1, 65), batch(2, 700)
    with native.World(small) as a, native.World(large) as b:
        a.snapshot()
        b.snapshot()
        want_a, want_b = gradients(a, small, 3, 2), gradients(b, large, 2, 1)
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        for _ in range(2):  # each in memory the other has left, b on a stream of the caller's
            for got, want in ((gradients(a, small, 3, 2), want_a), (gradients(b, large, 2, 1), want_b)):
                assert np.isfinite(want[0]).all()
                assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        b.set_stream(0)
        del stream
        b.rollout_record(1.0 / 60.0, 1, 1)  # frees and replaces the checkpoints used on that stream
        assert all(np.array_equal(x, y) for x, y in zip(gradients(a, small, 3, 2), want_a))
