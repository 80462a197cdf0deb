"""The substep's scan around the line between its two forms: up to 16,384 tiles
of 4,096 cells every block adds up the hash's tile sums before its own, above
that the blocks look back at one another.  Cell starts and occupancies against
the histogram of the sorted keys, over two substeps (the second scans the counts
and sums that the first one's force pass made).  1,019, 16,272
and 16,385 tiles."""
import pytest

from test_scan_gpu import test_scan_many_tiles as scan_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(161, 160, 161 + 1), (1023, 513, 127), (1024, 512, 128)])
def test_scan_forms(dims):
    # cells and one bucket: 4,173,121, 66,649,474 and 67,108,865
    scan_case(dims, 20000)
