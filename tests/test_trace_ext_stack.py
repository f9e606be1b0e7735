"""Callers' kernels (include/rdn_trace.cuh) whose parameters state a smaller stack than the walk needs: the pushes past
it are left out and set the context's error word, as parameters of another ordered walk or of an earlier build would."""

import ctypes as C
import struct

import numpy as np
import pytest

from helpers import Scene
from rendiation_gb300 import scenes
from test_trace_ext import MODE_WIDE4, build_extension

STACK_DEPTH = 4 * 8 + 5 * 4  # byte offset in the parameter block: four pointers and five words before it


@pytest.mark.gpu
@pytest.mark.parametrize("traversal", [0, 2])
def test_pushes_past_the_stated_depth(tmp_path, cuda, traversal):
    import torch

    lib = C.CDLL(build_extension(tmp_path))
    lib.trace_custom.argtypes = [C.c_void_p] * 3 + [C.c_uint32] * 5 + [C.c_void_p]
    mesh = scenes.heightfield(40, seed=7)
    P = Scene([[(mesh.positions, mesh.indices, 1)]], [[{"blas": 0}]]).build_product()
    rays = scenes.sphere_rays(3000, (0, 0, -0.2), (1, 1, 0.5), seed=3)
    d_rays = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    prm = []
    for t in (traversal, 2):
        size = C.c_size_t(0)
        assert P._L.rdn_trace_params(P._h, t, None, C.byref(size)) == 0
        buf = (C.c_uint8 * size.value)()
        assert P._L.rdn_trace_params(P._h, t, buf, C.byref(size)) == 0
        prm.append(buf)
    stated, needed = (struct.unpack_from("<I", b, STACK_DEPTH)[0] for b in prm)
    assert 8 < stated and 8 < needed <= 64

    def run(depth):
        b = (C.c_uint8 * len(prm[0])).from_buffer_copy(prm[0])
        struct.pack_into("<I", b, STACK_DEPTH, depth)
        out = torch.zeros((rays.shape[0], 4), device="cuda")
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.trace_custom(b, d_rays.data_ptr(), out.data_ptr(), rays.shape[0], 0, MODE_WIDE4, 0, 0xFF, s) == 0
        return out.cpu().numpy(), P.check_errors()

    whole, errors = run(needed)
    assert errors == (0, 0) and (whole[:, 3].view(np.uint32) != 0xFFFFFFFF).mean() > 0.2
    _, (status, word) = run(2)
    assert status != 0 and word & 1
    again, errors = run(needed)
    assert errors == (0, 0) and np.array_equal(whole.view(np.uint32), again.view(np.uint32))
