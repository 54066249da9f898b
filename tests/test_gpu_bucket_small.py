"""Sorts of a few thousand to half a million 32-bit keys: by buckets, or turned
away to the digit passes."""
import numpy as np
import pytest
import torch

import parallelalgorithms_gb300 as pa

pytestmark = pytest.mark.gpu
SIZES = [8191, 8192, 8193, 8200, 12_289, 65_535, 65_536, 262_145, 524_287, 524_288]


def _keys(kind, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    if kind == "sorted":
        keys.sort()
    elif kind == "narrow":
        keys = keys % np.uint32(5000) + np.uint32(77)
    elif kind == "clusters":
        keys = (keys >> np.uint32(30) << np.uint32(30)) + keys % np.uint32(n)
    elif kind == "constant":
        keys[:] = 42
    elif kind == "half constant":
        keys[rng.random(n) < 0.5] = 1 << 31
    elif kind == "outlier":
        keys = keys % np.uint32(1 << 16)
        keys[n // 3] = (1 << 32) - 1
    return keys


@pytest.mark.parametrize("kind", ["uniform", "sorted", "narrow", "clusters", "constant", "half constant", "outlier"])
@pytest.mark.parametrize("n", SIZES)
def test_keys(kind, n):
    keys = _keys(kind, n)
    d = torch.empty(n + 3, dtype=torch.int32, device="cuda")[n % 3:n % 3 + n]
    d.copy_(torch.from_numpy(keys.view(np.int32)))
    pa.sort(d.view(torch.uint32))
    assert np.array_equal(d.cpu().numpy().view(np.uint32), np.sort(keys))
