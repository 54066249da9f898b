"""Sorts of keys that repeat a pattern (records, rows of a matrix) whose period
divides the strides of the bucket plan's sample: right, and no longer than a few
times what evenly spread keys of the same number take (either sort is within a
factor of three; a bucket with most of the keys took some hundred times as long)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def structured(kind, n, torch):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int32)
    if kind == "pairs":  # a key and a flag by turns
        x[1::2] &= 3
    elif kind == "rows":  # one identifier and 63 small numbers a row
        y = x & 0xFFFF
        y[::64] = x[::64]
        x = y
    elif kind == "strides":  # only the first key of each stride is spread
        y = torch.arange(n, dtype=torch.int32, device="cuda") & 0xFFFFF
        at = (torch.arange(1 << 14, device="cuda") * n) >> 14
        y[at] = x[at]
        x = y
    return x


def timed_sort(pa, torch, src):
    best, keys, tmp = 1e9, torch.empty_like(src), torch.empty_like(src)
    for _ in range(3):
        keys.copy_(src)
        torch.cuda.synchronize()
        t = time.perf_counter()
        pa.sort(keys, tmp_keys=tmp)
        best = min(best, time.perf_counter() - t)
    return keys, best


@pytest.mark.parametrize("kind", ["pairs", "rows", "strides"])
@pytest.mark.parametrize("n", [1 << 20, 1 << 24, 1 << 26])
@pytest.mark.parametrize("wide", [False, True])
def test_period_of_a_stride(pa, torch_cuda, kind, n, wide):
    torch = torch_cuda
    if wide and n > 1 << 24:
        pytest.skip("one large size")

    def keys_of(k):
        x = structured(k, n, torch)
        return (x.to(torch.int64) << 32) | (structured("even", n, torch).to(torch.int64) & 0xFFFFFFFF) if wide else x

    _, even = timed_sort(pa, torch, keys_of("even"))
    src = keys_of(kind)
    got, took = timed_sort(pa, torch, src)
    flip = torch.iinfo(src.dtype).min
    assert torch.equal(got ^ flip, torch.sort(src ^ flip)[0])
    assert took < 10 * even, f"{took * 1e6:.0f} us against {even * 1e6:.0f}"


@pytest.mark.parametrize("kind", ["pairs", "rows"])
@pytest.mark.parametrize("share", [0.0, 0.2, 0.5, 0.9])
@pytest.mark.parametrize("n", [1 << 20, 1 << 26])
def test_select_of_a_pattern(pa, torch_cuda, kind, share, n):
    """The order statistic of such keys, in at most three times what evenly spread
    keys take: their sample brackets it as well."""
    torch = torch_cuda
    took = {}
    for k in ("even", kind):
        src = structured(k, n, torch)
        rank = int(n * share)
        want = int((torch.sort(src ^ -(1 << 31))[0][rank] ^ -(1 << 31)).item()) & 0xFFFFFFFF
        took[k] = 1e9
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            got = pa.select(src, rank)
            took[k] = min(took[k], time.perf_counter() - t)
        assert got == want
    assert took[kind] < 3 * took["even"], took
