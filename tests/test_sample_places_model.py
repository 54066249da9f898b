"""CPU model of the samples of bucket plans and selects (sample_place, csrc/pa_common.cuh): a place
in every stride, and every phase of a pattern that repeats seen in proportion."""
import numpy as np
import pytest


def places(log2, n):
    i = np.arange(1 << log2, dtype=np.uint64)
    lo, hi = (i * np.uint64(n)) >> np.uint64(log2), ((i + np.uint64(1)) * np.uint64(n)) >> np.uint64(log2)
    h = (i.astype(np.uint32) * np.uint32(0x9E3779B9)).astype(np.uint32)
    h = ((h ^ (h >> np.uint32(15))) * np.uint32(0x9E3779B9)).astype(np.uint32)
    h ^= h >> np.uint32(13)
    return lo, hi, lo + ((h.astype(np.uint64) * (hi - lo)) >> np.uint64(32))


@pytest.mark.parametrize("log2, n", [(14, 4097), (14, 8193), (14, 16384), (14, 100_003), (14, 100_663_296), (10, 4097),
                                     (10, 6_291_456)])
def test_in_their_strides(log2, n):
    lo, hi, at = places(log2, n)
    assert np.all(at >= lo) and np.all(at < np.maximum(hi, lo + np.uint64(1))) and int(at[-1]) < n


@pytest.mark.parametrize("log2, n", [(14, 1 << 20), (14, 1 << 24), (14, 1 << 26), (14, 100_000_000), (10, 1 << 20)])
@pytest.mark.parametrize("period", [2, 3, 4, 16, 64])
def test_phases_of_a_period(log2, n, period):
    seen = np.bincount((places(log2, n)[2] % np.uint64(period)).astype(np.int64), minlength=period)
    mean = (1 << log2) / period
    assert np.all(np.abs(seen - mean) < 6 * np.sqrt(mean))
