"""64-bit sorts by their leading digits: what the passes left out would have
ordered is mended, and payloads of equal keys keep their order."""
import numpy as np
import pytest
import torch

import parallelalgorithms_gb300 as pa

pytestmark = pytest.mark.gpu
LEAST = 1 << 19
M64 = (1 << 64) - 1


def _sampled(n):
    """Indices the device looks at before it leaves passes out."""
    lg = 12
    while lg < 17 and (1 << (2 * lg)) < 256 * n:
        lg += 1
    at = set()
    for i in range(1 << lg):
        g = (i + 1) * 0x9E3779B97F4A7C15 & M64
        at.add(((g * g & M64) ^ (g >> 29)) * n >> 64)
    return at


def _free(n, rng, count):
    """`count` places in increasing order that are not sampled."""
    hit = np.zeros(n, bool)
    hit[list(_sampled(n))] = True
    return np.sort(rng.choice(np.flatnonzero(~hit), count, replace=False))


def _groups(n, rng, keys, sizes, low_bits=32):
    """Groups of keys that agree above their low bits, at places not sampled."""
    at = rng.permutation(_free(n, rng, sum(sizes)))
    done = 0
    for size in sizes:
        top = np.uint64(int(rng.integers(1, 1 << (64 - low_bits))) << low_bits)
        low = rng.integers(0, 1 << low_bits, size, dtype=np.uint64)
        low[::3] = low[0]  # equal keys among them
        keys[at[done:done + size]] = top | low
        done += size


def _make(kind, n, seed):
    rng = np.random.default_rng(seed)
    keys = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if kind == "short":
        _groups(n, rng, keys, [2] * 300 + [3, 5, 31, 32])
    elif kind == "long":
        _groups(n, rng, keys, [32, 33, 34, 100, 511, 512, 513, 5000] + [40] * 50)
    elif kind == "ends":  # the groups' keys lie first and last
        keys[:] = (keys >> np.uint64(2)) + np.uint64(1 << 62)
        at = _free(n, rng, 80)
        keys[at[:40]] = rng.integers(0, 1 << 32, 40, dtype=np.uint64)
        keys[at[40:]] = np.uint64(0xFFFFFFFF << 32) | rng.integers(0, 1 << 32, 40, dtype=np.uint64)
        keys[at[79]] = np.uint64(M64)
    elif kind == "pairs":  # every other key has a neighbour it must change places with
        at = _free(n, rng, n // 4 * 2)
        keys[at[1::2]] = keys[at[::2]] & np.uint64(0xFFFFFFFF00000000)
        keys[at[::2]] |= np.uint64(1)
    elif kind == "many long":  # more long runs than are listed: every pass after all
        at = _free(n, rng, n // 64 * 40)
        keys[at] = rng.integers(1, n // 64, len(at), dtype=np.uint64) << np.uint64(32) | keys[at] & np.uint64(0xFFFFFFFF)
    elif kind == "too long":  # a run longer than one block mends: every pass after all
        at = _free(n, rng, (1 << 18) + 50)
        keys[at] = keys[at] & np.uint64(0xFFFFFFFF) | np.uint64(7 << 32)
    elif kind == "composite":  # a third of the range agrees in the leading digits
        keys = rng.integers(0, 1 << 10, n, dtype=np.uint64) << np.uint64(54) | keys & np.uint64((1 << 30) - 1)
    elif kind == "gap":  # bytes 2 and 6 hold one value
        keys = keys & np.uint64(0xFF00FFFFFF00FFFF) | np.uint64(0x0055000000AA0000)
        _groups(n, rng, keys, [], 32)
    elif kind == "six bytes":
        keys = keys & np.uint64((1 << 48) - 1)
        _groups(n, rng, keys, [2] * 50, 16)
        keys &= np.uint64((1 << 48) - 1)
    elif kind == "five bytes":
        keys = keys & np.uint64((1 << 40) - 1)
    elif kind == "ones":
        keys[rng.integers(0, n, n // 3)] = np.uint64(M64)
    return keys


KINDS = ["uniform", "short", "long", "ends", "pairs", "many long", "too long", "composite", "gap", "six bytes", "five bytes", "ones"]


@pytest.mark.parametrize("n", [LEAST - 1, LEAST, 600_011])
@pytest.mark.parametrize("kind", KINDS)
def test_pairs(kind, n):
    keys = _make(kind, n, 5)
    order = np.argsort(keys, kind="stable")
    k = torch.from_numpy(keys.copy().view(np.int64)).cuda().view(torch.uint64)
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    pa.sort(k, v)
    assert np.array_equal(k.cpu().numpy(), keys[order])
    assert np.array_equal(v.cpu().numpy(), order.astype(np.int32))


@pytest.mark.parametrize("kind", ["short", "long", "pairs", "too long"])
def test_large(kind):
    n = 20_000_003
    keys = _make(kind, n, 6)
    order = np.argsort(keys, kind="stable")
    k = torch.from_numpy(keys.copy().view(np.int64)).cuda().view(torch.uint64)
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    pa.sort(k, v)
    assert np.array_equal(k.cpu().numpy(), keys[order])
    assert np.array_equal(v.cpu().numpy(), order.astype(np.int32))


@pytest.mark.parametrize("kind", ["short", "long", "pairs", "too long"])
def test_keys_alone_that_crowd(kind):
    n = 900_001
    rng = np.random.default_rng(8)
    keys = _make(kind, n, 7)
    for value in keys[:3].copy():  # most keys are one of three
        keys[rng.integers(0, n, n // 3)] = value
    k = torch.from_numpy(keys.copy().view(np.int64)).cuda().view(torch.uint64)
    pa.sort(k)
    assert np.array_equal(k.cpu().numpy(), np.sort(keys))


@pytest.mark.parametrize("kind", ["short", "too long"])
def test_host_arrays(kind):
    n = 600_011
    keys = _make(kind, n, 9)
    order = np.argsort(keys, kind="stable")
    k, v = keys.copy(), np.arange(n, dtype=np.uint32)
    pa.sort(k, v)
    assert np.array_equal(k, keys[order])
    assert np.array_equal(v, order.astype(np.uint32))
