"""Batched plans that sort by buckets, against the oracle: segment sizes around
one bucket, around each count of buckets and tiles and around the longest
segment that is partitioned; segments whose keys crowd and are left to the digit
passes; buffers that start anywhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 5, 4095, 4096, 4097, 6143, 6144, 6145, 8191, 8192, 8193, 12288, 12289, 65537, 786_432, 786_433]
LONGEST = 2048 * 3072


def fill(kind, sizes, seed):
    rng = np.random.default_rng(seed)
    off = np.zeros(len(sizes) + 1, np.uint64)
    off[1:] = np.cumsum(np.asarray(sizes, np.uint64))
    keys = rng.integers(0, 1 << 32, int(off[-1]), dtype=np.uint32)
    if kind == "narrow":
        keys = keys % np.uint32(1 << 24) + np.uint32(1000)
    elif kind == "mixed":  # few values, in order, one heavy value, clusters, uniform by turns
        for i, (a, b) in enumerate(zip(off[:-1].astype(int), off[1:].astype(int))):
            if i % 5 == 0:
                keys[a:b] %= 7
            elif i % 5 == 1:
                keys[a:b] = np.arange(b - a)
            elif i % 5 == 2:
                keys[a:b:3] = 12345
            elif i % 5 == 3:
                keys[a:b] = (keys[a:b] // np.uint32(1 << 28) << np.uint32(28)) + keys[a:b] % np.uint32(50)
    elif kind == "skewed":
        keys = np.minimum(rng.random(keys.size) ** -1.5 * 1000, 2e9).astype(np.uint32)
    return keys, off


@pytest.mark.parametrize("kind", ["uniform", "narrow", "mixed", "skewed"])
@pytest.mark.parametrize("sizes", [EDGES, EDGES[::-1], [3000] * 40, [LONGEST, 7, LONGEST + 1, 20_000]],
                         ids=["edges", "edges_reversed", "whole", "longest"])
def test_plan(pa, port, torch_cuda, kind, sizes):
    from parallelalgorithms_gb300.batched import SegmentedSortPlan
    torch = torch_cuda
    keys, off = fill(kind, sizes, len(sizes))
    n = keys.size
    shift = 1 if len(sizes) == len(EDGES) else 0  # the array need not start at a 16-byte boundary
    buf = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    tmp = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    d, t = buf[shift:shift + n], tmp[2 * shift:2 * shift + n]
    plan = SegmentedSortPlan(off)
    for _ in range(2):  # the second run replays the graph over what the first one left in the plan
        d.copy_(torch.from_numpy(keys.view(np.int32)))
        plan.run(d, t)
    got = d.cpu().numpy().view(np.uint32)
    for i, (a, b) in enumerate(zip(off[:-1].astype(int), off[1:].astype(int))):
        want, _ = port.sort(keys[a:b])
        np.testing.assert_array_equal(got[a:b], want, err_msg=f"segment {i} [{a}, {b})")
    assert not buf[:shift].any() and not buf[shift + n:].any(), "keys outside the array were written"
    plan.close()
