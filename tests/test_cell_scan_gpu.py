"""The cell scan (kernels.cu) at its edges, seen through SpatialHash.query:
the queries' offsets are the scan of their counts, and query q sits on a
cluster of q % 7 points.  Rows of 128 counts to a warp, 512 a warp, 4,096 a
tile; more than 256 tiles take the prefix kernel."""
import numpy as np
import pytest

from blobs_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 2, 3, 4, 5, 127, 128, 129, 511, 513, 4095, 4096, 4097, 8191, 256 * 4096 - 1,
                                256 * 4096 + 1])
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
