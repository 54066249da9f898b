"""CPU model of the half of a bucket's cells that the count kernel lays out
(crowd_add, csrc/pa_buckets.cu): a place of its own for each entry, half of the
entries for every bucket, and multiples of any power of two in half of the buckets."""
import pytest

CELLS, ENTRIES, BUCKETS = 65536, 1024, 8


def place(cell, part):
    entry = (cell // 32) & (2 * ENTRIES - 1)
    return None if (bin(entry).count("1") ^ part) & 1 else entry // 2


@pytest.mark.parametrize("part", range(BUCKETS))
def test_places(part):
    seen = [place(32 * e, part) for e in range(2 * ENTRIES)]
    taken = [p for p in seen if p is not None]
    assert sorted(taken) == list(range(ENTRIES))
    assert all(place(32 * e + 31, part) == p for e, p in enumerate(seen))


@pytest.mark.parametrize("step", [32 << k for k in range(12)])
def test_multiples(step):
    for cell in range(0, CELLS, step):
        assert sum(place(cell, part) is not None for part in range(BUCKETS)) == BUCKETS // 2
