"""Keys-only sorts by buckets against the oracle: sizes around the least one,
around one and two partition passes and around tiles; key spreads that fill
buckets evenly, unevenly, with equal keys, with clusters, with a few keys far
outside, and that leave the sort to the digit passes; unaligned buffers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEAST_U32 = 1 << 19


def spread(name, n, bits, rng):
    full = 1 << bits
    dt = np.uint32 if bits == 32 else np.uint64
    if name == "uniform":
        return rng.integers(0, full, n, dtype=dt)
    if name == "narrow":  # the map starts above zero and ends well below the type's end
        return (rng.integers(0, 3 * n // 2, n, dtype=np.uint64) + full // 5).astype(dt)
    if name == "sorted":
        return (np.arange(n, dtype=np.uint64) + 77).astype(dt)
    if name == "heavy":  # two values hold about 2000 keys in a million each
        x = rng.integers(0, full, n, dtype=dt)
        x[rng.random(n) < 0.002] = full // 3
        x[rng.random(n) < 0.002] = full - 5
        return x
    if name == "copies":  # every value about 100 times
        return rng.integers(0, full, n // 100, dtype=dt)[rng.integers(0, n // 100, n)]
    if name == "clusters":  # about 150 keys within 16 values
        c = rng.integers(0, full - 16, n // 150, dtype=dt)
        return c[rng.integers(0, n // 150, n)] + rng.integers(0, 16, n, dtype=dt)
    if name == "outliers":  # nearly all keys in 2^18 values, a few at the type's ends
        x = (rng.integers(0, 1 << 18, n, dtype=np.uint64) + full // 2).astype(dt)
        x[n // 3], x[n // 2], x[7], x[n - 1] = 0, full - 1, 5, full - 2
        return x
    if name == "halves":  # one half of the keys in 1/8 of the range
        x = rng.integers(0, full, n, dtype=dt)
        x[::2] >>= dt(3)
        return x
    raise ValueError(name)


NAMES = ["uniform", "narrow", "sorted", "heavy", "copies", "clusters", "outliers", "halves"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("n", [LEAST_U32 - 1, LEAST_U32, 786_433, 3_000_001])
def test_u32(pa, port, name, n):
    a = spread(name, n, 32, np.random.default_rng(n))
    want, _ = port.sort(a)
    got = a.copy()
    pa.sort(got)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("n", [4097, 8193, 100_003, 786_433, 1_600_001])
def test_u64(pa, port, name, n):
    a = spread(name, n, 64, np.random.default_rng(n))
    want, _ = port.sort(a)
    got = a.copy()
    pa.sort(got)
    np.testing.assert_array_equal(got, want)


SMALL = [1, 2, 3, 31, 511, 512, 513, 2047, 4095, 4096, 4097, 8191, 8192]


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("kind", ["uniform", "constant", "few", "sorted", "pairs", "outlier", "offset"])
def test_few_keys(pa, port, torch_cuda, bits, kind):
    """Whole sorts by one CTA: every size at which its steps change, in place on
    a buffer that need not start at a 16-byte boundary."""
    dt, signed = (np.uint32, np.int32) if bits == 32 else (np.uint64, np.int64)
    rng = np.random.default_rng(bits)
    for n in SMALL:
        a = rng.integers(0, 1 << bits, n, dtype=dt)
        if kind == "constant":
            a[:] = a[0]
        elif kind == "few":
            a = a[rng.integers(0, min(n, 5), n)]
        elif kind == "sorted":
            a = np.arange(n, dtype=dt)
        elif kind == "pairs":  # every value twice: one collision each
            a[n // 2:2 * (n // 2)] = a[:n // 2]
        elif kind == "outlier":
            a %= dt(1000)
            a[n // 2] = dt((1 << bits) - 1)
        want, _ = port.sort(a)
        skip = 1 if kind == "offset" else 0
        buf = torch_cuda.zeros(n + 8, dtype=torch_cuda.int32 if bits == 32 else torch_cuda.int64, device="cuda")
        keys = buf[skip:skip + n]
        keys.copy_(torch_cuda.from_numpy(a.view(signed)))
        pa.sort(keys)
        np.testing.assert_array_equal(keys.cpu().numpy().view(dt), want, err_msg=f"n = {n}")
        assert not buf[:skip].any() and not buf[skip + n:].any()


@pytest.mark.parametrize("n", SMALL)
def test_few_floats(pa, port, n):
    a = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint32)
    a[:n // 3] = np.random.default_rng(n).standard_normal(n // 3).astype(np.float32).view(np.uint32)
    flip = lambda b: b ^ np.where(b >> 31, 0xFFFFFFFF, 0x80000000).astype(np.uint32)  # noqa: E731
    want, _ = port.sort(flip(a))
    got = a.view(np.float32).copy()
    pa.sort(got)
    np.testing.assert_array_equal(flip(got.view(np.uint32)), want)


@pytest.mark.parametrize("kind", ["range", "normal", "signs"])
def test_f32(pa, port, kind):
    rng = np.random.default_rng(7)
    n = LEAST_U32 + 12345
    if kind == "range":  # spread as evenly as floats of one binade are
        a = (1.0 + rng.random(n)).astype(np.float32)
    elif kind == "normal":
        a = rng.standard_normal(n).astype(np.float32)
    else:
        a = rng.integers(0, 1 << 32, n, dtype=np.uint32).view(np.float32)  # NaNs of every payload among them
    want, _ = port.sort(a.view(np.uint32) ^ np.where(a.view(np.uint32) >> 31, 0xFFFFFFFF, 0x80000000).astype(np.uint32))
    got = a.copy()
    pa.sort(got)
    bits = got.view(np.uint32)
    np.testing.assert_array_equal(bits ^ np.where(bits >> 31, 0xFFFFFFFF, 0x80000000).astype(np.uint32), want)


@pytest.mark.parametrize("offset, tmp_offset", [(0, 1), (1, 0), (1, 2), (3, 3)])
@pytest.mark.parametrize("bits, n", [(32, LEAST_U32 + 5), (64, 50_001)])
def test_unaligned_buffers(pa, port, torch_cuda, bits, n, offset, tmp_offset):
    torch = torch_cuda
    a = spread("uniform", n, bits, np.random.default_rng(offset))
    want, _ = port.sort(a)
    signed = torch.int32 if bits == 32 else torch.int64
    buf = torch.zeros(n + 8, dtype=signed, device="cuda")
    tmp = torch.zeros(n + 8, dtype=signed, device="cuda")
    keys = buf[offset:offset + n]
    keys.copy_(torch.from_numpy(a.view(np.int32 if bits == 32 else np.int64)))
    pa.sort(keys, tmp_keys=tmp[tmp_offset:tmp_offset + n])
    np.testing.assert_array_equal(keys.cpu().numpy().view(a.dtype), want)
    assert not buf[:offset].any() and not buf[offset + n:].any(), "keys outside the array were written"
    assert not tmp[:tmp_offset].any() and not tmp[tmp_offset + n:].any(), "scratch outside the array was written"
