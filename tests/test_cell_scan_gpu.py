"""The cell scan (kernels.cu) at its edges, seen through SpatialHash.query:
the queries' offsets are the scan of their counts, and query q sits on a
cluster of q % 7 points.  One block up to 16,384 counts, in rows of 128;
beyond, tiles of 4,096, 512 a warp; more than 256 tiles take the prefix
kernel."""
import numpy as np
import pytest

from blobs_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 2, 3, 4, 5, 127, 128, 129, 511, 513, 4095, 4096, 4097, 8191, 16383, 16384,
                                16385, 16386, 20_481, 256 * 4096 - 1, 256 * 4096 + 1])
def test_offsets_of_known_counts(nq):
    centre = np.stack([np.arange(7) * 10.0, np.zeros(7)], 1).astype(np.float32)
    which = np.repeat(np.arange(7), np.arange(7))
    with native.SpatialHash(1.0) as h:
        h.set_points(np.arange(len(which), dtype=np.uint64) * 3 + 1, centre[which], np.full(len(which), 0.1, np.float32))
        q = np.arange(nq) % 7
        offsets, ids = h.query(centre[q], np.full(nq, 0.2, np.float32))
    assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(q)]).astype(np.uint64))
    first = np.concatenate([[0], np.cumsum(np.arange(7))])
    want = [first[k] + np.arange(k) for k in range(7)]
    some = min(nq, 5000)
    assert np.array_equal(ids[:int(offsets[some])], np.concatenate([want[k] for k in q[:some]]) * 3 + 1)


@pytest.mark.parametrize("per_cell", [1, 7, 8, 33, 200])
def test_query_result_sizes(per_cell):
    """Results of one query below, at and above the sizes its lanes rank
    themselves (64), from one cell and from all nine, ids in any order."""
    rng = np.random.Generator(np.random.PCG64(per_cell))
    gx, gy = np.meshgrid(np.arange(12), np.arange(12))
    centre = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.float32) + 0.5
    xy = (np.repeat(centre, per_cell, 0) + rng.uniform(-0.45, 0.45, (144 * per_cell, 2))).astype(np.float32)
    ids = rng.permutation(len(xy) * 3)[:len(xy)].astype(np.uint64)
    radius = rng.uniform(0.0, 0.2, len(xy)).astype(np.float32)
    qxy = np.concatenate([centre, rng.uniform(-2.0, 14.0, (201, 2)).astype(np.float32)])
    qr = rng.choice(np.array([0.0, 0.3, 1.0, 5.0], np.float32), len(qxy))
    with native.SpatialHash(1.0) as h:
        h.set_points(ids, xy, radius)
        offsets, got = h.query(qxy, qr)
        exact = h.query(qxy, qr, cap=len(got))
    assert np.array_equal(exact[0], offsets) and np.array_equal(exact[1], got)
    cell, qcell = np.floor(xy).astype(int), np.floor(qxy).astype(int)
    for k in range(len(qxy)):
        near = (np.abs(cell - qcell[k]) <= 1).all(1)
        e = xy - qxy[k]
        d = (qr[k] + radius).astype(np.float32)
        hit = near & ((e[:, 0] * e[:, 0]) + (e[:, 1] * e[:, 1]) <= d * d)
        assert np.array_equal(got[int(offsets[k]):int(offsets[k + 1])], np.sort(ids[hit]))
