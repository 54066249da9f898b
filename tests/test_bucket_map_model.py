"""CPU model of the bucket map: monotone, every bucket's least key as the
finish kernel computes it, and the cells and bins of a bucket within bounds."""
import random

import pytest

CELLS, BINS = 65536, 4096


def make_map(lo, hi, bits, nb):
    """The map the plan kernel lays over a sample spanning [lo, hi]."""
    top = (1 << bits) - 1
    pad = (hi - lo) >> 10
    lo -= min(lo, pad)
    hi += min(top - hi, pad)
    if hi - lo >= (top >> 3) * 7:
        lo, hi = 0, top
    s = max(0, (hi - lo).bit_length() - 32) if bits == 64 else 0
    rng = ((hi - lo) >> s) + 1
    mult = min((nb << 32) // rng, (1 << 32) - 1)
    width = ((1 << 32) + mult - 1) // mult
    sh = 0
    while ((width - 1) >> sh) >= CELLS:
        sh += 1
    cell = sh + s
    while ((width - 1) >> sh) >= BINS:
        sh += 1
    return {"lo": lo, "s": s, "mult": mult, "inv": (1 << 63) // mult, "cell": cell, "bin": sh + s, "nb": nb}


def bucket(m, key):
    t = min(max(key - m["lo"], 0) >> m["s"], (1 << 32) - 1)
    return min((t * m["mult"]) >> 32, m["nb"] - 1)


def first_t(m, b):
    t = ((b << 33) * m["inv"]) >> 64
    steps = 0
    while (t * m["mult"]) >> 32 < b:
        t += 1
        steps += 1
    assert steps <= 2
    return t


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("nb", [256, 512, 4096, 32768])
def test_map(bits, nb):
    r = random.Random(bits * nb)
    top = (1 << bits) - 1
    spans = [(0, top), (0, 0), (5, 5), (top, top), (0, nb - 2), (3, nb + 3), (0, 100_000_000), (top - 3 * nb, top),
             (top // 3, top // 3 + 12345), (0, top // 8 * 7), (0, top // 8 * 7 - 1000)]
    spans += [tuple(sorted((r.randrange(top), r.randrange(top)))) for _ in range(20)]
    for lo, hi in spans:
        m = make_map(lo, hi, bits, nb)
        for b in [1, 2, nb // 2, nb - 2] + [r.randrange(1, nb - 1) for _ in range(20)]:
            t0, t1 = first_t(m, b), first_t(m, b + 1)
            if t0 >= 1 << 32:
                continue
            least = m["lo"] + (t0 << m["s"])
            if least > top:
                continue
            # the least key of the bucket, and none below it belongs to it
            if t0 < t1:
                assert bucket(m, least) == b
            if t0 > 0:
                assert bucket(m, m["lo"] + (t0 << m["s"]) - 1) < b
            if t0 < t1:  # every key of the bucket falls in a cell and a bin
                greatest = min(m["lo"] + (t1 << m["s"]) - 1, top)
                assert bucket(m, greatest) == b
                assert (greatest - least) >> m["cell"] < CELLS
                assert (greatest - least) >> m["bin"] < BINS
        keys = sorted([r.randrange(top + 1) for _ in range(200)] + [0, top, lo, hi])
        where = [bucket(m, k) for k in keys]
        assert where == sorted(where) and 0 <= where[0] and where[-1] < nb
