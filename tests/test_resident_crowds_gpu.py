"""Small worlds whose bodies have many candidates -- a large body among small
ones, a box or circle too small for its bodies -- run by the kernels of a
substep, those that stay sparse by whole steps in one launch (k_resident), and
either way with the same states as phase by phase."""
import numpy as np
import pytest

from blobs_gb300 import native, scenes
from test_resident_gpu import check, single

pytestmark = pytest.mark.gpu


def one_large(n, factor, seed=0):
    """n spheres of radius 0.05 to 0.15 at 60% packing, one of them of factor * 0.15."""
    rng = np.random.Generator(np.random.PCG64(100 * n + seed))
    rad = rng.uniform(0.05, 0.15, n).astype(np.float32)
    rad[n // 2] = np.float32(0.15 * factor)
    half = np.float32(np.sqrt(np.pi * float((rad.astype(np.float64) ** 2).sum()) / 0.6) / 2 + rad.max())
    s = scenes.spheres(rng.uniform(-half, half, (n, 2)).astype(np.float32), rad,
                       rng.normal(0.0, 0.5, (n, 2)).astype(np.float32))
    s.world_box = np.array([[-half, -half, half, half]], np.float32)
    s.dt = 1.0 / 120.0
    return s


@pytest.mark.parametrize("n,factor,resident", [(2000, 1.5, True), (2000, 2.0, False), (500, 6.0, False), (500, 1.5, True),
                                               (257, 2.0, False), (256, 2.0, True), (256, 3.0, False), (96, 8.0, True),
                                               (97, 20.0, False), (2, 30.0, True)])
def test_one_large_body(n, factor, resident):
    check(one_large(n, factor), steps=2, resident=resident)


def test_a_batch_with_one_crowded_world():
    for factor, resident in ((1.0, True), (5.0, False)):
        s = scenes.pack([single(200 + k, 0.35, seed=k) for k in range(5)] + [one_large(700, factor)])
        s.dt = 1.0 / 120.0
        check(s, steps=2, resident=resident)


@pytest.mark.parametrize("n,packing,resident", [(1000, 3.0, True), (1000, 5.0, False), (90, 5.0, True)])
def test_overfilled_boxes(n, packing, resident):
    check(single(n, packing), steps=2, resident=resident)


@pytest.mark.parametrize("radius,resident", [(4.0, True), (1.0, False)])
def test_overfilled_circles(radius, resident):
    s = single(600, 0.3)
    s.circles = np.array([[0.0, 0.0, radius], [0.0, 0.0, 50.0]], np.float32)
    check(s, steps=2, resident=resident)


def test_cells_wider_than_the_bodies():
    """A large cell size from the configuration crowds any world."""
    s = single(600, 0.4)
    for cell_size, resident in ((0.0, True), (3.0, False)):
        with native.World(s, cell_size=cell_size) as w:
            before = w.kernel_launches()
            w.step(s.dt)
            assert (w.kernel_launches() - before < 10) == resident
