"""The algorithmic bytes reported for a batch's filter programs are those of the forms the device reads."""
import pytest

import rhydb_gpu as R
from rawtable import RawBuilder

pytestmark = pytest.mark.gpu


def test_bytes_of_a_coverage_leaf():
    late = "N" * 9 + "A" * 119  # covered from position 10 on
    inside = "A" * 19 + "N" * 10 + "A" * 99  # a missing interval of 4 bytes in the position's block
    b = RawBuilder(6).add_sequences("main", 0, "A" * 128, [late, inside, inside, inside, "A" * 128, late])
    raw = b.raw()
    dev = R.Device(R.Table.from_raw(raw), 0)
    for position, bounds in ((5, 2), (50, 0)):  # 8 bytes per row whose covered region misses the position
        dev.batch_prepare([f"SymEq(main,{position},N)"])
        assert dev.batch_info().filter_bytes == 8 + 8 * bounds + 4 * 3  # the count, the bounds, the intervals
    dev.close()
