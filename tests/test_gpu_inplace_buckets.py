"""The in-place sort's groups, sorted by buckets where their digits are evenly
filled: even, uneven, and crowded inside their digits."""
import numpy as np
import pytest
import torch

import parallelalgorithms_gb300 as pa

pytestmark = pytest.mark.gpu


def _keys(kind, n, rng):
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    if kind == "half range":  # the upper 128 digits are empty
        keys >>= np.uint32(1)
    elif kind == "uneven":
        keys = (rng.random(n) ** 3 * (1 << 32)).astype(np.uint64).clip(0, (1 << 32) - 1).astype(np.uint32)
    elif kind == "crowded inside":  # even digits, few values in each
        keys &= np.uint32(0xFF000007)
    elif kind == "gaps":  # every third digit is empty
        keys = np.where((keys >> np.uint32(24)) % 3 == 0, keys ^ np.uint32(1 << 24), keys)
    elif kind == "sorted":
        keys.sort()
    return keys


@pytest.mark.parametrize("kind", ["even", "half range", "uneven", "crowded inside", "gaps", "sorted"])
@pytest.mark.parametrize("n,scratch", [(600_001, 0), (3_000_017, 700_000), (3_000_017, 1 << 16)])
def test_groups(kind, n, scratch):
    keys = _keys(kind, n, np.random.default_rng(n + scratch))
    d = torch.from_numpy(keys.view(np.int32).copy()).cuda().view(torch.uint32)
    pa.parallel_hybrid_inplace_msd_radix_sort(d, scratch_keys=scratch)
    assert np.array_equal(d.cpu().numpy(), np.sort(keys))
