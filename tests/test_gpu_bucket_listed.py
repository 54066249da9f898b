"""Bucket sorts where most buckets are left to the launch behind the finish
kernel, many buckets to a CTA: keys that crowd into two clusters of each bucket,
a value of each bucket that repeats, buckets counted by value whose range is wide
because of a few keys far away."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crowd(kind, n, bits, bucket_bits, rng):
    """n keys spread evenly over 1 << bucket_bits buckets of the key's top bits."""
    dt = np.uint32 if bits == 32 else np.uint64
    width = bits - bucket_bits
    top = rng.integers(0, 1 << bucket_bits, n, dtype=dt) << dt(width)
    if kind == "clusters":
        return top + (rng.integers(0, 2, n, dtype=dt) << dt(width - 1)) + rng.integers(0, 1000, n, dtype=dt)
    x = top + rng.integers(0, 1 << width, n, dtype=dt)  # repeats: one key in 200 is its bucket's own value
    some = rng.random(n) < 0.005
    x[some] = top[some] + dt(12345)
    return x


def by_package(pa, torch, keys):
    d = torch.from_numpy(keys.view(np.int32 if keys.dtype == np.uint32 else np.int64).copy()).cuda()
    pa.sort(d)
    return d.cpu().numpy().view(keys.dtype)


@pytest.mark.parametrize("kind", ["clusters", "repeats"])
@pytest.mark.parametrize("bits, n, bucket_bits", [(32, 20_000_003, 13), (64, 6_000_001, 11), (32, 700_001, 8)])
def test_most_buckets_listed(pa, torch_cuda, kind, bits, n, bucket_bits):
    keys = crowd(kind, n, bits, bucket_bits, np.random.default_rng(n))
    assert np.array_equal(by_package(pa, torch_cuda, keys), np.sort(keys))


@pytest.mark.parametrize("bits, n", [(32, 20_000_003), (64, 6_000_001)])
def test_counted_with_far_keys(pa, torch_cuda, bits, n):
    rng = np.random.default_rng(bits)
    keys = rng.integers(1 << 28, (1 << 28) + 4 * n, n, dtype=np.uint64).astype(np.uint32 if bits == 32 else np.uint64)
    keys[[7, n // 3, n // 2 + 1, n - 2]] = [0, (1 << bits) - 1, 5, (1 << bits) - 2]
    assert np.array_equal(by_package(pa, torch_cuda, keys), np.sort(keys))


@pytest.mark.parametrize("kind", ["clusters", "repeats", "far"])
def test_batched(pa, torch_cuda, kind):
    from parallelalgorithms_gb300.batched import SegmentedSortPlan
    torch = torch_cuda
    rng = np.random.default_rng(len(kind))
    segments, size = 300, 65_537
    off = np.arange(segments + 1, dtype=np.uint64) * size
    if kind == "far":  # counted: 32 buckets of at most 8192 values, and both end buckets wide
        keys = rng.integers(1 << 28, (1 << 28) + (1 << 17), segments * size, dtype=np.uint32)
        keys[off[:-1].astype(np.int64) + 33] = 1
        keys[off[1:].astype(np.int64) - 44] = (1 << 32) - 2
    else:
        keys = crowd(kind, segments * size, 32, 5, rng)
    d = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    plan = SegmentedSortPlan(off)
    plan.run(d, torch.empty_like(d))
    plan.close()
    got = d.cpu().numpy().view(np.uint32).reshape(segments, size)
    assert np.array_equal(got, np.sort(keys.reshape(segments, size), axis=1))
