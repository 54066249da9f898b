"""Digit passes run by a grid of resident CTAs that loop over tiles: key +
payload sorts whose tiles are just fewer than, as many as and just more than
the resident CTAs, and twice as many, against numpy's stable order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (keys per tile, CTAs per SM) of the key + payload passes
GEOMETRY = {np.uint32: (512 * 12, 2), np.uint64: (256 * 12, 3)}


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("times, extra", [(1, -1), (1, 0), (1, 1), (2, 0), (2, 1)])
def test_tiles_around_the_resident_grid(dtype, times, extra):
    import torch

    import parallelalgorithms_gb300 as pa
    tile, per_sm = GEOMETRY[dtype]
    grid = torch.cuda.get_device_properties(0).multi_processor_count * per_sm
    n = times * grid * tile + extra
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 20, n, dtype=dtype)  # equal keys: the order of the payloads matters
    order = np.argsort(keys, kind="stable")
    signed = np.int32 if dtype is np.uint32 else np.int64
    k = torch.from_numpy(keys.view(signed)).cuda()
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    pa.sort(k, v)
    np.testing.assert_array_equal(v.cpu().numpy(), order.astype(np.int32))
    np.testing.assert_array_equal(k.cpu().numpy().view(dtype), keys[order])
