"""Bucket sorts of keys that repeat: buckets of few values are counted, wider
ones left to the digit passes; keys outside the sampled range."""
import numpy as np
import pytest
import torch

import parallelalgorithms_gb300 as pa
from parallelalgorithms_gb300 import batched

pytestmark = pytest.mark.gpu
SPAN = 8192  # values of a counted bucket, at most


def _keys(n, span, low, rng):
    return (rng.integers(0, span, n, dtype=np.uint64) + low).astype(np.uint32)


def _sorted(keys):
    d = torch.from_numpy(keys.view(np.int32).copy()).cuda().view(torch.uint32)
    pa.sort(d)
    return d.cpu().numpy()


@pytest.mark.parametrize("low", [0, 123_457, (1 << 32) - (1 << 30)])
@pytest.mark.parametrize("span", [1000, 65535, 70_000, 256 * SPAN - 5000, 256 * SPAN, 256 * SPAN + 5000, 512 * SPAN, 1 << 24, 1 << 30])
@pytest.mark.parametrize("n", [600_011, 700_000])
def test_narrow_ranges(n, span, low):
    keys = _keys(n, span, low, np.random.default_rng(span))
    assert np.array_equal(_sorted(keys), np.sort(keys))


@pytest.mark.parametrize("span", [1 << 16, 1 << 20, 1 << 27, 1 << 28])
def test_two_partitions(span):
    keys = _keys(20_000_003, span, 77, np.random.default_rng(span))
    assert np.array_equal(_sorted(keys), np.sort(keys))


@pytest.mark.parametrize("span", [3000, 1 << 20, 256 * SPAN - 9, 256 * SPAN + 9999, 1 << 23, 1 << 40])
@pytest.mark.parametrize("n", [500_009, 6_000_011])
def test_long_keys(n, span):
    rng = np.random.default_rng(n + span)
    keys = rng.integers(0, span, n, dtype=np.uint64) + np.uint64(1 << 50)
    keys[3] = np.uint64(5)
    d = torch.from_numpy(keys.view(np.int64).copy()).cuda().view(torch.uint64)
    pa.sort(d)
    assert np.array_equal(d.cpu().numpy(), np.sort(keys))


def test_outliers_and_frequent_values():
    rng = np.random.default_rng(3)
    keys = _keys(1_000_003, 1 << 20, 1 << 21, rng)
    keys[[5, 77, 900_001]] = [0, (1 << 32) - 1, 1 << 31]  # not sampled: the end buckets' range is wide
    keys[rng.integers(0, keys.size, 6000)] = (1 << 21) + 500_000  # one bucket beyond shared memory
    assert np.array_equal(_sorted(keys), np.sort(keys))


@pytest.mark.parametrize("span", [50, 4096, 100_000, 1 << 20, 1 << 23])
def test_batched(span):
    rng = np.random.default_rng(span)
    sizes = np.array([100_000, 3, 50_001, 4097, 1_000_000, 0, 250_007])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    keys = _keys(int(off[-1]), span, 99, rng)
    d = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    plan = batched.SegmentedSortPlan(off)
    plan.run(d, torch.empty_like(d))
    got = d.cpu().numpy().view(np.uint32)
    for a, b in zip(off[:-1].astype(int), off[1:].astype(int)):
        assert np.array_equal(got[a:b], np.sort(keys[a:b]))
