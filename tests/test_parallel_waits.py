"""The look-back kernels of the scan, the compaction and the sort when a tile before them never publishes: their waits
run out, they count that tile in the input themselves, and what they write is right (whole numbers, all equal).
tests/parallel_waits.cu launches the kernels with the first tiles left out; nothing waits without a limit."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from helpers import ROOT

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
UNTOUCHED = 0x5A5A5A5A


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("waits") / "libwaits.so")
    cmd = [NVCC, "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_103a,code=sm_103a",
           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "rendiation_gb300", "csrc"),
           os.path.join(ROOT, "tests", "parallel_waits.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    p, u = C.c_void_p, C.c_uint32
    L.waits_scan.argtypes = [p, p, u, u, C.c_int, C.c_int, u, p]
    L.waits_compact.argtypes = [p, p, p, p, u, u, p]
    L.waits_sort.argtypes = [p, p, p, p, u, u, u, C.c_int, p]
    return L


def test_waits_compile(lib):
    assert lib.waits_tile(0) == 8192 and lib.waits_tile(1) == 4096


def device(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32).copy()).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("tiles,tail,skip", [(2, 1, 1), (3, 8192, 2), (40, 77, 1), (40, 8192, 35)])
@pytest.mark.parametrize("form", ["exclusive", "inclusive flags", "in place", "misaligned", "segments"])
def test_scan(lib, cuda, tiles, tail, skip, form):
    import torch

    tile = lib.waits_tile(0)
    n = (tiles - 1) * tile + tail
    x = np.random.default_rng(n).integers(0, 2**32, n, dtype=np.uint32)
    if "flags" in form:
        x[x % 3 == 0] = 0
    d = device(np.concatenate([np.zeros(1, np.uint32), x])) if form == "misaligned" else device(x)
    at = d.data_ptr() + (4 if form == "misaligned" else 0)
    out = torch.full((n,), UNTOUCHED, dtype=torch.int32, device="cuda")
    dst = at if form == "in place" else out.data_ptr()
    scratch = torch.zeros(64 + 8 * tiles, dtype=torch.uint8, device="cuda")
    inclusive = form in ("inclusive flags", "segments")
    segment = 4 if form == "segments" else 0
    assert lib.waits_scan(at, dst, n, skip, inclusive, "flags" in form, segment, scratch.data_ptr()) == 0
    got = (d if form == "in place" else out).cpu().numpy().view(np.uint32)
    v = (x != 0).astype(np.uint32) if "flags" in form else x
    want = np.cumsum(v, dtype=np.uint32)
    if segment:
        want = np.concatenate([np.cumsum(c, dtype=np.uint32) for c in np.split(v, range(4 * tile, n, 4 * tile))])
    if not inclusive:
        want -= v
    assert np.array_equal(got[skip * tile:], want[skip * tile:])
    assert np.array_equal(got[:skip * tile], x[:skip * tile] if form == "in place" else np.full(skip * tile, UNTOUCHED))


@pytest.mark.gpu
@pytest.mark.parametrize("tiles,tail,skip", [(2, 1, 1), (5, 8192, 3), (36, 500, 1)])
def test_compact(lib, cuda, tiles, tail, skip):
    import torch

    tile = lib.waits_tile(0)
    n = (tiles - 1) * tile + tail
    rng = np.random.default_rng(n)
    values, flags = rng.integers(0, 2**32, n, dtype=np.uint32), rng.integers(0, 3, n, dtype=np.uint32)
    dv, df = device(values), device(flags)
    out = torch.full((n,), UNTOUCHED, dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(64 + 8 * tiles, dtype=torch.uint8, device="cuda")
    assert lib.waits_compact(dv.data_ptr(), df.data_ptr(), out.data_ptr(), count.data_ptr(), n, skip, scratch.data_ptr()) == 0
    keep = flags != 0
    left_out = int(keep[:skip * tile].sum())
    got = out.cpu().numpy().view(np.uint32)
    assert int(count) == keep.sum()
    assert np.array_equal(got[left_out:keep.sum()], values[keep][left_out:])
    assert np.all(got[:left_out] == UNTOUCHED) and np.all(got[keep.sum():] == UNTOUCHED)


@pytest.mark.gpu
@pytest.mark.parametrize("tiles,tail,skip", [(2, 1, 1), (7, 4096, 6), (20, 33, 2)])
@pytest.mark.parametrize("wide,shift", [(0, 0), (0, 24), (1, 8)])
def test_sort_pass(lib, cuda, tiles, tail, skip, wide, shift):
    import torch

    tile = lib.waits_tile(1)
    n = (tiles - 1) * tile + tail
    keys = np.random.default_rng(n).integers(0, 2**32, n, dtype=np.uint32)
    keys[: n // 3] &= np.uint32(0x07070707)  # digits with long runs
    dk, dv = device(keys), device(np.arange(n, dtype=np.uint32))
    ok, ov = (torch.full((n,), UNTOUCHED, dtype=torch.int32, device="cuda") for _ in range(2))
    scratch = torch.zeros(16 * 256 + 256 + tiles * 256 * 8, dtype=torch.uint8, device="cuda")
    assert lib.waits_sort(dk.data_ptr(), dv.data_ptr(), ok.data_ptr(), ov.data_ptr(), n, shift, skip, wide,
                          scratch.data_ptr()) == 0
    order = np.argsort((keys >> np.uint32(shift)) & np.uint32(255), kind="stable")
    written = order >= skip * tile
    gk, gv = ok.cpu().numpy().view(np.uint32), ov.cpu().numpy().view(np.uint32)
    assert np.array_equal(gk[written], keys[order[written]]) and np.array_equal(gv[written], order[written])
    assert np.all(gk[~written] == UNTOUCHED)
