"""CPU model of the flags of the bucket sort's finish loop (finish_buckets,
csrc/pa_buckets.cu): a CTA's warps read the counters of one bucket, which decide
what barriers they take part in, and thread 0 clears them for the next bucket.
Interleavings of two warps over a few buckets are tried (all with up to
MOST_SWITCHES forced switches): each warp must take the branch that its bucket asks
for, and both must always wait at the same barrier."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parents[1] / "parallelalgorithms_gb300" / "csrc" / "pa_buckets.cu"
MOST_SWITCHES = 3


def warp(me, buckets, flags, order, barrier):
    """One warp's steps; yields the barrier it waits at, or None after a step."""
    for b, kind in enumerate(buckets):
        if me == 0:  # thread 0's warp
            flags["nhit"] = flags["over"] = 0
            yield None
        yield ("top", b)
        crowded = kind == "crowded"
        if crowded:  # keys that find their cell taken: every warp adds to the counter
            flags["nhit"] += 1
            yield None
        if kind == "entry" and me == 1:
            flags["nhit"] = 1
            yield None
        yield ("hits", b)
        nhit = flags["nhit"]
        yield None
        listed = nhit > 1
        if nhit and not listed:
            if me == 1 and kind == "entry":
                flags["over"] = 1
                yield None
            yield ("turns", b)
            listed = flags["over"] != 0
            yield None
        order[me].append(listed)
        if not listed:
            yield ("scan", b)
            yield ("out", b)
        elif barrier:
            yield ("listed", b)


def sound(buckets, barrier):
    """Whether the interleavings take the right branches and pair up their barriers."""
    want = [k != "even" for k in buckets]

    def play(schedule):
        """Runs a schedule (which warp makes each step, as far as it is given);
        returns the choices there were, or False for a mismatch."""
        flags, order = {"nhit": 0, "over": 0}, [[], []]
        run = [warp(0, buckets, flags, order, barrier), warp(1, buckets, flags, order, barrier)]
        at, ended, choices = [None, None], [False, False], []
        while not all(ended):
            ready = [w for w in (0, 1) if not ended[w] and at[w] is None]
            if not ready:
                if any(ended) or at[0] != at[1]:
                    return False
                at = [None, None]
                continue
            pick = schedule[len(choices)] if len(choices) < len(schedule) else ready[0]
            if pick not in ready:
                pick = ready[0]
            choices.append((pick, len(ready)))
            try:
                at[pick] = next(run[pick])
            except StopIteration:
                ended[pick] = True
                other = 1 - pick
                if not ended[other] and at[other] is not None:
                    return False
        return choices if order[0] == want and order[1] == want else False

    todo = [([], 0)]
    while todo:
        schedule, switches = todo.pop()
        choices = play(schedule)
        if choices is False:
            return False
        for i in range(len(schedule), len(choices)):
            if choices[i][1] == 2 and switches < MOST_SWITCHES:
                todo.append(([c for c, _ in choices[:i]] + [1 - choices[i][0]], switches + 1))
    return True


@pytest.mark.parametrize("buckets", [["crowded", "even"], ["entry", "even"], ["crowded", "entry", "even"], ["even", "even"]])
def test_barrier_behind_a_listed_bucket(buckets):
    assert sound(buckets, barrier=True)
    if buckets[0] != "even":
        assert not sound(buckets, barrier=False), "without the barrier some interleaving goes wrong"


def test_source_has_the_barrier():
    body = SOURCE.read_text().split("finish_buckets(uint32_t nb", 1)[1]
    listing = re.search(r"if \(!done[^\n]*\n?.*?rare\[1 \+ atomicAdd\(rare, 1u\)\] = job\.number;(.*?)\n  }\n", body, re.S)
    assert listing and "__syncthreads();" in listing.group(1)
