"""Select by a bracket and its even bins: what one block narrows, what is left
to the digit steps, and inputs that are their own sample; waiting and
asynchronous calls alike."""
import ctypes

import numpy as np
import pytest
import torch

import parallelalgorithms_gb300 as pa
from parallelalgorithms_gb300 import _native

pytestmark = pytest.mark.gpu


def _inputs(n, dtype, rng):
    top = np.iinfo(dtype).max
    full = rng.integers(0, top, n, dtype=dtype, endpoint=True)
    mid = full.copy()  # all but a few keys within a narrow range in the middle: one full bin
    where = rng.random(n) < 0.97
    mid[where] = top // 2 + rng.integers(0, 1000, int(where.sum()), dtype=dtype)
    few = rng.integers(0, 7, n, dtype=dtype) * dtype(top // 7)
    pairs = full.copy()
    pairs[n // 2:n // 2 * 2] = pairs[:n // 2]
    ends = np.where(rng.random(n) < 0.5, dtype(0), dtype(top))
    return {
        "full": full,
        "narrow": rng.integers(5, 1500, n, dtype=dtype),
        "sorted": np.sort(full),
        "crowded": mid,
        "few": few,
        "pairs": pairs,
        "ends": ends.astype(dtype),
        "top": np.full(n, top, dtype),
    }


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("n", [1, 2, 8191, 8192, 8193, 40_003, 3_000_001])
def test_ranks(n, dtype):
    rng = np.random.default_rng(n)
    kind = "u32" if dtype == np.uint32 else "u64"
    for name, a in _inputs(n, dtype, rng).items():
        want = np.sort(a)
        d = torch.from_numpy(a.view(np.int32 if dtype == np.uint32 else np.int64)).cuda()
        d = d.view(torch.uint32 if dtype == np.uint32 else torch.uint64)
        out = torch.zeros(1, dtype=torch.int64, device="cuda")
        for k in sorted({0, 1 % n, n // 3, n // 2, max(0, n - 2), n - 1}):
            assert pa.select(d, k) == want[k], (name, k)
            stream = torch.cuda.current_stream()
            _native.call(f"pa_select_{kind}", ctypes.c_void_p(d.data_ptr()), n, k, ctypes.c_void_p(out.data_ptr()),
                         _native.opts(stream.cuda_stream, async_device=True))
            torch.cuda.synchronize()
            assert out.cpu().numpy().view(dtype)[0] == want[k], (name, k)
