"""Bucket sorts of keys that fill their buckets evenly and crowd into few cells of
each: multiples of a number, few prefixes with small numbers behind them, clusters,
a value of each bucket that repeats.  Right, and turned away to the digit passes
before they move: left to the launch for listed buckets they take up to seven times
what evenly spread keys take."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crowded(kind, n, wide, torch):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64)
    low = torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64)
    if kind == "even":
        y = (x << 32) | low if wide else x
    elif kind == "multiples":
        y = (x >> 8) << 40 if wide else x // 1000 * 1000
    elif kind == "prefixes":  # 2^20 of them, and small numbers
        y = ((x & 0xFFFFF) << 40) | low if wide else ((x & 0xFFFFF) << 12) | (low & 15)
    elif kind == "clusters":  # 16 values around each of n / 150 places
        c = torch.randint(0, 1 << 31, (n // 150,), generator=g, device="cuda", dtype=torch.int64) << (32 if wide else 1)
        y = c[torch.randint(0, n // 150, (n,), generator=g, device="cuda")] + (low & 15)
    elif kind == "repeats":  # one key in 40 is one of 2^17 values
        v = torch.randint(0, 1 << 32, (1 << 17,), generator=g, device="cuda", dtype=torch.int64)
        y = torch.where(low % 40 == 0, v[low & 0x1FFFF], x)
        y = y << 32 if wide else y
    return y if wide else (y - ((y >> 31) << 32)).to(torch.int32)


def asynchronous(pa, torch, keys, tmp):
    from parallelalgorithms_gb300 import _native
    o = _native.PaOpts()
    o.async_device = 1
    name = "pa_sort_u32" if keys.dtype == torch.int32 else "pa_sort_u64"
    _native.call(name, keys.data_ptr(), tmp.data_ptr(), keys.numel(), ctypes.pointer(o))


def best_of(f, restore, torch, times=4):
    best = 1e9
    for _ in range(times):
        restore()
        torch.cuda.synchronize()
        t = time.perf_counter()
        f()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("waits", [True, False])
@pytest.mark.parametrize("kind", ["multiples", "prefixes", "clusters", "repeats"])
@pytest.mark.parametrize("wide, n", [(False, 1 << 26), (True, (1 << 24) + 1)])
def test_whole_arrays(pa, torch_cuda, kind, wide, n, waits):
    torch = torch_cuda
    took = {}
    for k in ("even", kind):
        src = crowded(k, n, wide, torch)
        keys, tmp = src.clone(), torch.empty_like(src)
        run = (lambda: pa.sort(keys, tmp_keys=tmp)) if waits else (lambda: asynchronous(pa, torch, keys, tmp))
        took[k] = best_of(run, lambda: keys.copy_(src), torch)
        flip = torch.iinfo(src.dtype).min
        assert torch.equal(keys ^ flip, torch.sort(src ^ flip)[0])
    # (by digit passes: 1.7 and 3.1 times)
    assert took[kind] < (4.5 if wide else 2.5) * took["even"], took


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("kind", ["multiples", "clusters", "repeats"])
@pytest.mark.parametrize("shift", [0, 1])
def test_least_sizes_and_places(pa, torch_cuda, kind, wide, shift):
    """Around the least size that is looked at, scratch that starts anywhere."""
    torch = torch_cuda
    least = 1 << (20 if wide else 21)
    for n in (least - 1, least, least + 3):
        src = crowded(kind, n, wide, torch)
        keys = src.clone()
        tmp = torch.empty(n + 4, dtype=src.dtype, device="cuda")
        pa.sort(keys, tmp_keys=tmp[shift:shift + n])
        flip = torch.iinfo(src.dtype).min
        assert torch.equal(keys ^ flip, torch.sort(src ^ flip)[0])


@pytest.mark.parametrize("kind", ["multiples", "prefixes", "clusters", "repeats"])
@pytest.mark.parametrize("size", [4097, 6145, 100_001, 1_000_003])
def test_batched(pa, torch_cuda, kind, size):
    from parallelalgorithms_gb300.batched import SegmentedSortPlan
    torch = torch_cuda
    segments = max(4, 20_000_000 // size)
    off = np.arange(segments + 1, dtype=np.uint64) * size
    plan = SegmentedSortPlan(off)
    took = {}
    for k in ("even", kind):
        src = crowded(k, segments * size, False, torch)
        if k == "clusters":  # each segment's own: 16 values around each of size / 150 places
            c = src.view(segments, size)[:, :size // 150].contiguous()
            at = torch.randint(0, size // 150, (segments, size), device="cuda")
            src = (torch.gather(c, 1, at) + torch.randint(0, 16, (segments, size), device="cuda", dtype=torch.int32)).view(-1)
        d, t = torch.empty_like(src), torch.empty_like(src)
        took[k] = best_of(lambda: plan.run(d, t), lambda: d.copy_(src), torch)
        flip = -(1 << 31)
        want = torch.sort((src ^ flip).view(segments, size), dim=1)[0].view(-1)
        assert torch.equal(d ^ flip, want)
    plan.close()
    assert took[kind] < 3.2 * took["even"], took
