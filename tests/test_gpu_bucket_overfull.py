"""Bucket sorts whose sample looks even though buckets hold more keys than the
finish kernel: the exact counts turn them away before a key is moved.  Waiting and
asynchronous calls, in-place groups, and the sizes from which an asynchronous call
has both sorts enqueued."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def comb(n, bits, bucket_bits, share, torch, seed=1):
    """Keys in every 1/share-th bucket (of the top bucket_bits) alone: no part of
    the range looks full, but these buckets hold 1/share times the mean."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    used = int((1 << bucket_bits) * share)
    top = (torch.randint(0, used, (n,), generator=g, device="cuda", dtype=torch.int64) / share).to(torch.int64)
    low = torch.randint(0, 1 << (32 - bucket_bits), (n,), generator=g, device="cuda", dtype=torch.int64)
    key = (top << (32 - bucket_bits)) | low
    if bits == 32:
        return (key - ((key >> 31) << 32)).to(torch.int32)
    return (key << 32) | torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64)


def cluster(n, bits, size, torch):
    """Evenly spread keys with `size` of them in one bucket."""
    g = torch.Generator(device="cuda").manual_seed(n)
    dtype = torch.int32 if bits == 32 else torch.int64
    x = torch.randint(-(1 << (bits - 1)), (1 << (bits - 1)) - 1, (n,), generator=g, device="cuda", dtype=dtype)
    at = torch.randperm(n, generator=g, device="cuda")[:size]
    x[at] = torch.randint(1 << (bits - 3), (1 << (bits - 3)) + 30_000, (size,), generator=g, device="cuda", dtype=dtype)
    return x


def expect(torch, x):
    flip = torch.iinfo(x.dtype).min
    return torch.sort(x ^ flip)[0] ^ flip


def asynchronous(keys, tmp, torch):
    from parallelalgorithms_gb300 import _native
    o = _native.PaOpts()
    o.async_device = 1
    name = "pa_sort_u32" if keys.dtype == torch.int32 else "pa_sort_u64"
    _native.call(name, keys.data_ptr(), tmp.data_ptr(), keys.numel(), ctypes.pointer(o))
    torch.cuda.synchronize()


@pytest.mark.parametrize("bits", [32, 64])
def test_one_bucket(pa, torch_cuda, bits):
    """12,000 keys of 6M in one bucket: 33 of the sample, where 45 may be."""
    torch = torch_cuda
    src = cluster(6_000_001, bits, 12_000, torch)
    keys = src.clone()
    pa.sort(keys, tmp_keys=torch.empty_like(keys))
    assert torch.equal(keys, expect(torch, src))


@pytest.mark.parametrize("n, scratch", [(6_000_001, 0), (24_000_001, 6_200_000)])
def test_in_place(pa, torch_cuda, n, scratch):
    torch = torch_cuda
    src = cluster(n, 32, 12_000, torch)
    if scratch:  # in several groups
        src[::3000] = torch.randint(40 << 24, (40 << 24) + 30_000, (src[::3000].numel(),), device="cuda", dtype=torch.int32)
        src[1::3000] = torch.randint(-(100 << 24), -(100 << 24) + 30_000, (src[1::3000].numel(),), device="cuda", dtype=torch.int32)
    keys = src.clone()
    pa.parallel_hybrid_inplace_msd_radix_sort(keys, scratch_keys=scratch)
    assert torch.equal(keys, expect(torch, src))
    host = src.cpu().numpy().view(np.uint32).copy()
    pa.parallel_hybrid_inplace_msd_radix_sort(host, scratch_keys=scratch)
    assert np.array_equal(host, np.sort(src.cpu().numpy().view(np.uint32)))


SPREADS = [(32, (1 << 26) + 1, 15, 1 / 3), (64, 25_000_001, 13, 1 / 1.6)]


@pytest.mark.parametrize("bits, n, bucket_bits, share", SPREADS)
@pytest.mark.parametrize("kind", ["even", "comb", "crowded"])
@pytest.mark.parametrize("waits", [True, False])
def test_large(pa, torch_cuda, bits, n, bucket_bits, share, kind, waits):
    torch = torch_cuda
    src = comb(n, bits, bucket_bits, share if kind == "comb" else 1.0, torch)
    if kind == "crowded":  # the plan says no
        src[src < 0] = 77
    keys, tmp = src.clone(), torch.empty_like(src)
    if waits:
        pa.sort(keys, tmp_keys=tmp)
    else:
        asynchronous(keys, tmp, torch)
    assert torch.equal(keys, expect(torch, src))


@pytest.mark.parametrize("share", [1 / 3, 3 / 4])
def test_takes_no_longer_than_by_digits(pa, torch_cuda, share):
    """At most 2.5 times what evenly spread keys take: 1.7 by digit passes, 3.5 and
    more with every bucket left to the launch behind.  3/4: two parts of the range,
    three quarters of the keys in one, which the plan sees."""
    torch = torch_cuda
    n = 1 << 26 if share == 1 / 3 else 100_000_000
    best = {}
    for kind in ("even", "uneven"):
        if kind == "uneven" and share == 3 / 4:
            src = comb(n, 32, 15, 1.0, torch)
            src[n // 4 * 2:] &= 0x7FFFFFFF
        else:
            src = comb(n, 32, 15, share if kind == "uneven" else 1.0, torch)
        keys, tmp = torch.empty_like(src), torch.empty_like(src)
        best[kind] = 1e9
        for _ in range(4):
            keys.copy_(src)
            torch.cuda.synchronize()
            t = time.perf_counter()
            pa.sort(keys, tmp_keys=tmp)
            best[kind] = min(best[kind], time.perf_counter() - t)
        assert torch.equal(keys, expect(torch, src))
    assert best["uneven"] < 2.5 * best["even"], best
