"""The rebuild's scans at the edges of their accesses: element counts around
the eight items of a thread and the 2,048 of a tile, so that the last thread's
items are a whole access, a part of one or none.  The pair list follows from
all five scanned arrays and is compared with the FP64 oracle's, bit-exact."""
import pytest

from test_rebuild_edges import _box, _same_list

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 8, 9, 2039, 2040, 2046, 2047, 2048, 2049, 4095])   # n + 1 items are scanned
@pytest.mark.parametrize("levels", [1, 3])
def test_counts_around_an_access_and_a_tile(n, levels):
    assert _same_list(_box(n, 40 + n, levels), "f64") >= 0
