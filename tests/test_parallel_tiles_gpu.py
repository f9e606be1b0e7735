"""rdn_scan_u32, rdn_compact_u32 and rdn_radix_sort_u32 where their tiles of 4096
and 8192 elements begin, end and follow one another, against numpy (whole numbers:
no tolerance)."""

import ctypes as C

import numpy as np
import pytest

from rendiation_gb300 import native

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 4095, 4096, 4097, 8191, 8192, 8193, 16_385, 131_071, 135_169, 1_048_577]


def scratch(kind, n):
    """A block of exactly the size the library asks for, filled with ones."""
    import torch

    size = C.c_size_t()
    assert getattr(native.lib(), f"rdn_{kind}_scratch_size")(n, C.byref(size)) == 0
    buf = torch.full((size.value + 512,), 255, dtype=torch.uint8, device="cuda")
    return buf, (buf.data_ptr() + 255) & ~255, size.value


def array(x, skew=0):
    """x on the device, `skew` words past a 16-byte boundary."""
    import torch

    buf = torch.zeros(x.shape[0] + skew + 4, dtype=torch.int32, device="cuda")
    view = buf[skew:skew + x.shape[0]]
    view.copy_(torch.from_numpy(x.astype(np.uint32).view(np.int32)))
    return buf, view


def host(t):
    return t.cpu().numpy().view(np.uint32)


def guard(keep, size, ptr):
    """Nothing past the queried scratch was written."""
    off = ptr - keep.data_ptr() + size
    assert bool((keep[off:] == 255).all())


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_scan(cuda, n, skew):
    x = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)  # sums wrap
    inc = np.cumsum(x, dtype=np.uint32)
    for inclusive in (0, 1):
        for in_place in (False, True):
            _, d = array(x, skew)
            _, out = (None, d) if in_place else array(np.zeros(n, np.uint32), skew)
            keep, ptr, size = scratch("scan", n)
            assert native.lib().rdn_scan_u32(d.data_ptr(), out.data_ptr(), n, inclusive, 0, ptr, size, None) == 0
            assert np.array_equal(host(out), inc if inclusive else inc - x)
            guard(keep, size, ptr)


@pytest.mark.parametrize("segment", [1, 2, 32, 2048, 4096, 8192, 1 << 18, 1 << 30])
def test_segments(cuda, segment):
    n = 300_001
    x = np.random.default_rng(segment).integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    _, d = array(x)
    _, out = array(np.zeros(n, np.uint32))
    keep, ptr, size = scratch("scan", n)
    assert native.lib().rdn_scan_u32(d.data_ptr(), out.data_ptr(), n, 1, segment, ptr, size, None) == 0
    want = np.concatenate([np.cumsum(x[i:i + segment], dtype=np.uint32) for i in range(0, n, segment)]) \
        if segment > 1 else x
    assert np.array_equal(host(out), want)


@pytest.mark.parametrize("skew", [0, 3])
@pytest.mark.parametrize("share", [0.0, 0.001, 0.5, 1.0])
@pytest.mark.parametrize("n", SIZES)
def test_compaction(cuda, n, share, skew):
    import torch

    rng = np.random.default_rng(n)
    v = rng.integers(1, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    f = np.where(rng.random(n) < share, rng.integers(1, 1 << 32, n, dtype=np.uint64), 0).astype(np.uint32)
    _, dv = array(v, skew)
    _, df = array(f, 0)
    _, out = array(np.full(n, 9, np.uint32), skew)
    count = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    keep, ptr, size = scratch("compact", n)
    assert native.lib().rdn_compact_u32(dv.data_ptr(), df.data_ptr(), out.data_ptr(), count.data_ptr(), n, ptr, size,
                                        None) == 0
    kept = v[f != 0]
    assert int(count.item()) == kept.shape[0]
    assert np.array_equal(host(out), np.concatenate([kept, np.zeros(n - kept.shape[0], np.uint32)]))
    guard(keep, size, ptr)


@pytest.mark.parametrize("kind", ["random", "equal", "few", "high"])
@pytest.mark.parametrize("n", SIZES)
def test_sort(cuda, n, kind):
    rng = np.random.default_rng(n)
    for bits in (1, 8, 9, 17, 32):
        keys = rng.integers(0, 1 << bits, n, dtype=np.uint64)
        if kind == "equal":
            keys[:] = (1 << bits) - 1
        elif kind == "few":
            keys = keys % 3
        elif kind == "high":  # the lowest digit says nothing
            keys &= ~np.uint64(0xFF)
        keys = keys.astype(np.uint32)
        order = np.argsort(keys, kind="stable")
        for with_values in (True, False):
            _, dk = array(keys, 1)
            _, dv = array(np.arange(n, dtype=np.uint32), 2)
            keep, ptr, size = scratch("radix_sort", n)
            assert native.lib().rdn_radix_sort_u32(dk.data_ptr(), dv.data_ptr() if with_values else None, n, bits, ptr,
                                                   size, None) == 0
            assert np.array_equal(host(dk), keys[order])
            assert np.array_equal(host(dv), order if with_values else np.arange(n))
            guard(keep, size, ptr)
