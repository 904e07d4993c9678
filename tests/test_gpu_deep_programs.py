"""Programs whose counters need more stack tiles than a 4,096-row tile's shared memory holds: they run at 2,048 rows,
and the depth that is refused does not depend on it."""
import numpy as np
import pytest

import rhydb_gpu as R
from rawtable import oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def table():
    t = R.Table.generate(70000, seed=23, genome_len=900, pool_sites=300, null_fraction=0.01)
    dev = R.Device(t, 0)
    yield t, dev, oracle_for(t)
    dev.close()


def nested(t, levels):
    """NOf of 2 over four children, the last of them nested: two planes a level in the reference's counting, three on
    the device (a sticky one)."""
    pos, _, _, card, _ = t.containers(0)
    rows = {int(p): int(card[pos == p].sum()) for p in np.unique(pos)}
    dense = sorted(rows, key=lambda p: -rows[p])[:40]
    site = lambda i: f"HasMut(main,{dense[i % 40] + 1})"
    q = f"Or({site(0)},{site(1)})"
    for i in range(levels):
        q = f"NOf(2,{('atleast', 'exactly')[i % 2]},{site(i)},Not({site(i + 7)}),{site(3 * i + 2)},{q})"
    return q


@pytest.mark.parametrize("levels", [120, 134, 150, 195])  # 400 tiles of 4,096 rows fit
def test_programs_past_the_narrowest_schedule_width(table, levels):
    t, dev, orc = table
    q = nested(t, levels)
    obits, on = orc.compute_filter(q)
    bits, n = dev.compute_filter(q)
    assert n == on and np.array_equal(bits, obits)
    assert dev.count(q) == on
    short = [nested(t, 3), "HasMut(main,9)"]
    assert dev.batch([q, *short])[0].tolist() == [on, *(orc.count(x) for x in short)]
    counts, filtered = dev.mutations(q, 0)
    want, wn = orc.mutations(q, 0)
    assert filtered == wn and np.array_equal(counts, want)


def test_refused_depth_is_that_of_the_plain_program(table):
    t, dev, _ = table
    for call in (dev.count, lambda q: dev.batch([q])):
        with pytest.raises(R.IllegalQuery):
            call(nested(t, 201))
