"""The cell scan around the count up to which one block does it (8,192, two
rows of 128 a warp), as tests/test_cell_scan_gpu.py checks its other edges."""
import pytest

import test_cell_scan_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [4098, 8064, 8065, 8190, 8192, 8193, 8194, 8195])
def test_offsets_around_the_line(nq):
    test_cell_scan_gpu.test_offsets_of_known_counts(nq)
