"""Steps on a stream that the caller is capturing are refused before anything
is queued or changed, the capture stays valid, and the world goes on as if
the call had not been made."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def spheres(n):
    s = scenes.random_world(np.random.Generator(np.random.PCG64(n)), n, 0.05, 0.15, 0.5, 0.7)
    s.dt = 1.0 / 60.0
    return s


WORLDS = {
    "resident": lambda: spheres(700),
    "resident classes": lambda: scenes.pack([spheres(n) for n in (40, 300, 900)]),
    "spheres": lambda: spheres(5000),
    "jointed": lambda: scenes.jointed_bodies(seed=4, n=900, n_joints=200, n_springs=200, side=45.0),
}


def state(w):
    b = w.read_bodies()
    return [b[k] for k in ("pos", "pos_old", "vel", "rotation", "angvel")] + [w.read_snapshots(),
                                                                             np.array(w.contact_count()), np.array(w.time())]


@pytest.mark.parametrize("name", list(WORLDS))
def test_refused_under_capture(name):
    import torch
    s = WORLDS[name]()
    dt = 1.0 / 60.0
    stream = torch.cuda.Stream()
    x = torch.zeros(4, device="cuda")
    with native.World(s) as w, native.World(s) as plain:
        w.set_stream(stream.cuda_stream)
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream, capture_error_mode="relaxed"):
            x.add_(1.0)
            with pytest.raises(native.BlobsError):
                w.rollout(dt, 2)  # of a fresh world: its first step is irregular, the second not
        for k in range(3):  # a step's first, second and later uses
            w.step(dt)
            plain.step(dt)
            calls = [lambda: w.step(dt), lambda: w.rollout(dt, 3), lambda: w.fixed_step(dt)]
            if name != "jointed":
                calls.append(lambda: w.rollout_record(dt, 2, 1))
            launches = w.kernel_launches()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
                x.add_(1.0)
                for call in calls:
                    with pytest.raises(native.BlobsError):
                        call()
            assert w.kernel_launches() == launches
            graph.replay()
            torch.cuda.synchronize()
            assert x.tolist() == [1.0 + k] * 4
            for a, b in zip(state(w), state(plain)):
                assert np.array_equal(a, b)
        for f in (w, plain):
            f.rollout(dt, 3)
            f.fixed_step(dt)
        for a, b in zip(state(w), state(plain)):
            assert np.array_equal(a, b)
        w.set_stream(0)
