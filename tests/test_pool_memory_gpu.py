"""The memory that rollouts keep for the next call goes back to the device with
the device's last world, and not before: checked in a process of its own, so
that no other world or cache is in the way."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GB = 1 << 30


def check():
    import torch

    from blobs_gb300 import native, scenes

    def free_bytes():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    s = scenes.random_world(np.random.Generator(np.random.PCG64(1)), 100_000, 0.1, 0.2, 0.3, 1.0)
    s.dt = 1.0 / 60.0
    with native.World(s) as w:
        w.step(s.dt)
    before = free_bytes()
    for again in range(2):
        with native.World(s) as w:
            with native.World(s) as other:
                # 92 bytes per body and substep of a segment, and the checkpoints: over 3 GB
                other.rollout_record(s.dt, 45, 45)
                other.backward(np.ones((s.n_bodies, 2), np.float32), s.n_springs)
            assert before - free_bytes() > 3 * GB
            w.rollout_record(s.dt, 2, 1)  # its recording is open when the world goes
        assert before - free_bytes() < GB // 4


@pytest.mark.gpu
def test_kept_memory_goes_with_the_last_world():
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    check()
