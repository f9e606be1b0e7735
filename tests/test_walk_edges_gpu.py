"""Batches at the largest sizes that four lanes per ray are given, and trees so deep that no stack in local memory holds
their walks, against the reference order: the same results, except where a ray meets two triangles at exactly the same
distance."""

import ctypes as C
import struct

import numpy as np
import pytest

from helpers import Scene, rt, scenes
from rendiation_gb300 import native
from test_instanced_walks_gpu import params_tail

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def large(cuda):
    """A soup whose rays walk so much that every size rule is at its upper end; three of four camera rays hit it."""
    m = scenes.triangle_soup(20_000, seed=8, offset=0.05)
    P = Scene([[(m.positions, None, 1)]], [[{"blas": 0}]]).build_product(device_build=True)
    assert params_tail(P)[2] > 70  # quad_limit: 90 * 70^2 is above 400,000
    return P


def cuda_rays(rays):
    import torch

    return torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()


def trace(P, d, traversal, **kw):
    import torch

    hits = torch.full((d.shape[0], 4), -7.0, device="cuda")
    ext = torch.full((d.shape[0], 4), -7, dtype=torch.int32, device="cuda")
    P.trace(d, hits, ext, traversal=traversal, **kw)
    return np.concatenate([hits.cpu().numpy().view(np.int32), ext.cpu().numpy()], 1)


def assert_traces(P, d, watertight=0, **kw):
    want = trace(P, d, rt.TRAVERSAL_REFERENCE | watertight, **kw)
    for traversal in (rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        got = trace(P, d, traversal | watertight, **kw)
        differ = (got != want).any(1)
        assert np.count_nonzero(differ) <= d.shape[0] // 20_000
        # a tie: a hit on both sides, at the same distance
        assert np.array_equal(got[differ, 0], want[differ, 0]) and (want[differ, 3] != -1).all()
    return want


@pytest.mark.parametrize("n", [39_999, 40_001, 99_999, 100_033, 399_999, 400_001, 400_033])
def test_query_counts(large, n):
    cam = scenes.pinhole_rays(scenes.soup_camera(512, -(-n // 512)))[:n]
    rnd = scenes.sphere_rays(n, (-0.02,) * 3, (1.02,) * 3, seed=n)
    want = assert_traces(large, cuda_rays(np.where(((np.arange(n) + 16) // 96) % 2 == 0, cam, rnd)))
    assert (want[:, 3] != -1).mean() > 0.3


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("width,height", [(440, 450), (544, 544), (548, 548), (600, 504)])
def test_wavefront_frames(large, width, height, watertight):
    """198,000, 295,936, 300,304 and 302,400 pixels: secondary rays above 400,000 by quads, and both kinds of primaries."""
    import torch

    out = []
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
        wf = rt.Wavefront(large, scenes.soup_camera(width, height), (0.2, 0.2, 2.0))
        wf.configure((traversal | watertight, 64, 1), (traversal | watertight, 64, 1))
        wf.run(3)
        torch.cuda.synchronize()
        out.append((wf.results().copy().view(np.uint32).reshape(-1, 8), wf.rays_traced()))
    assert np.count_nonzero((out[0][0] != out[1][0]).any(-1)) <= width * height // 20_000
    assert out[0][1] == out[1][1]


@pytest.mark.parametrize("width,height", [(440, 448), (448, 456)])
def test_rendered_frames(large, width, height):
    """197,120 and 204,288 pixels."""
    import torch

    from rendiation_gb300 import path_tracing as pt
    from rendiation_gb300 import task_graph as tg

    eye = (0.5, -1.2, 1.1)
    vp = tg.look_at_view_projection_inv(eye, (0.5, 0.5, 0.5), (0, 0, 1), 40.0, width / height)
    lights = [pt.directional_light((3.0, 2.5, 2.0), (0.3, 0.2, -1.0))]
    out = []
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
        ao = tg.AmbientOcclusion(large, width, height, vp, eye, traversal=traversal)
        ao.render()
        R = pt.DeviceReferencePathTracingRenderer(large, width, height, vp, eye, lights=lights, traversal=traversal)
        R.render()
        torch.cuda.synchronize()
        out.append((ao.result().copy(), R.result().copy()))
    for a, b in zip(*out):
        assert np.count_nonzero((a != b).any(-1)) <= width * height // 20_000


# ---- deep trees -----------------------------------------------------------------------------------------------------

DEEP, RATIO = 30, 0.45


def deep_mesh(levels, seed):
    """Clusters of 16 triangles, each 0.45 of the one before in size and distance from the origin. A node's other
    child is smaller than the cluster beside it, so the four-child nodes open the clusters and keep a level for each."""
    rng = np.random.default_rng(seed)
    tri = []
    for k in range(levels):
        s = RATIO**k
        c = s * (0.3 + 0.7 * rng.random((16, 1, 3)))
        tri.append(c + s * rng.uniform(-0.25, 0.25, (16, 3, 3)))
    return np.concatenate(tri).astype(np.float32).reshape(-1, 3)


@pytest.fixture(scope="module")
def deep(cuda):
    P = Scene([[(deep_mesh(DEEP, 5), None, 1)]], [[{"blas": 0}]], blas_bin_size=1).build_product(device_build=True, blas_max_depth=64)
    size = C.c_size_t(0)
    assert P._L.rdn_trace_params(P._h, 1, None, C.byref(size)) == 0
    buf = (C.c_uint8 * size.value)()
    assert P._L.rdn_trace_params(P._h, 1, buf, C.byref(size)) == 0
    entries = struct.unpack_from("<I", bytes(buf), 4 * 8 + 6 * 4)[0]  # of a four-child walk's stack
    assert entries > 64, entries
    return P


def deep_rays(n, seed):
    """Rays through the clusters of every size, from all sides and from the origin outwards (not through the origin from
    afar, where distances to the clusters around it are alike to the last bit)."""
    rng = np.random.default_rng(seed)
    s = RATIO ** rng.integers(0, DEEP, n)[:, None]
    at = s * (0.4 + 0.7 * rng.random((n, 3)))
    d = rng.normal(size=(n, 3))
    org = at - 2 * s * d / np.linalg.norm(d, axis=1, keepdims=True)
    d[::6], org[::6] = at[::6], 0.0
    return scenes.make_rays(org.astype(np.float32), d.astype(np.float32))


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("n,local", [(900, 0), (900, 1), (50_000, 1), (410_001, 0), (410_001, 1)])
def test_deep_queries(deep, n, local, watertight):
    want = assert_traces(deep, cuda_rays(deep_rays(n, n)), watertight, local_stack=local)
    assert (want[:, 3] != -1).mean() > 0.2 and deep.check_errors() == (0, 0)


@pytest.mark.parametrize("refill", [0, 8])
@pytest.mark.parametrize("n", [3000, 420_000])
def test_deep_paths(deep, n, refill):
    import torch

    d = cuda_rays(deep_rays(n, n))
    out = []
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        p = rt.Paths(deep, d, max_bounces=2, seed=7, traversal=traversal, refill=refill if traversal != 1 else 0)
        p.run()
        torch.cuda.synchronize()
        out.append(p.results().copy())
    for got in out[1:]:
        assert np.count_nonzero(got != out[0]) <= n // 20_000
    assert deep.check_errors() == (0, 0)


@pytest.mark.parametrize("n", [500, 160_000, 410_001])
def test_deep_differentiable(deep, n):
    import torch

    d = cuda_rays(deep_rays(n, n))
    attr = torch.rand(48 * DEEP, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    out = []
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
        z = lambda *s, dtype=torch.float32: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
        tri, hit, seg = z(n, dtype=torch.int32), z(n, 4), z(n, 2, dtype=torch.int32)
        h = native.HitDiffDesc(rays=d.data_ptr(), count=n, attributes=attr.data_ptr(), traversal=traversal,
                               hit=hit.data_ptr(), hit_tri=tri.data_ptr())
        p = native.AttrPathDesc(rays=d.data_ptr(), count=n, segments=2, seed=3, attributes=attr.data_ptr(),
                                grad_scale=1.0, traversal=traversal, seg_tri=seg.data_ptr())
        assert native.lib().rdn_hit_diff_forward(deep._h, C.byref(h), None) == 0
        assert native.lib().rdn_attr_paths_forward(deep._h, C.byref(p), None) == 0
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (tri, hit, seg)])
    same = out[0][0] == out[1][0]
    assert np.count_nonzero(~same) <= n // 20_000
    assert np.array_equal(out[0][1][same], out[1][1][same], equal_nan=True)
    assert np.count_nonzero((out[0][2] != out[1][2]).any(1)) <= n // 20_000
    assert deep.check_errors() == (0, 0)


@pytest.mark.parametrize("width,height", [(120, 90), (560, 560)])
def test_deep_frames(deep, width, height):
    import torch

    from rendiation_gb300 import path_tracing as pt
    from rendiation_gb300 import task_graph as tg

    eye = (1.6, 1.4, 1.5)
    vp = tg.look_at_view_projection_inv(eye, (0.2, 0.2, 0.2), (0, 0, 1), 40.0, width / height)
    cam = scenes.PinholeCamera.look_at(eye, (0.2, 0.2, 0.2), 40.0, width, height)
    lights = [pt.directional_light((3.0, 2.5, 2.0), (-0.3, -0.2, -1.0))]
    out = []
    for traversal, refill in ((rt.TRAVERSAL_REFERENCE, 0), (rt.TRAVERSAL_ORDERED, 0), (rt.TRAVERSAL_ORDERED_WIDE, 8)):
        wf = rt.Wavefront(deep, cam, (0.2, 0.2, 2.0))
        wf.configure((traversal, 64, 0), (traversal, 64, 0), refill=refill)
        wf.run(3)
        ao = tg.AmbientOcclusion(deep, width, height, vp, eye, traversal=traversal)
        ao.render()
        graph = tg.AmbientOcclusion(deep, width, height, vp, eye, traversal=traversal, mode="graph")
        graph.render()
        images = [wf.results().copy().view(np.uint32).reshape(-1, 8), ao.result().copy(), graph.result().copy()]
        for schedule in (0, 1, 2):
            R = pt.DeviceReferencePathTracingRenderer(deep, width, height, vp, eye, lights=lights, traversal=traversal,
                                                      schedule=schedule)
            R.render()
            images.append(R.result().copy())
        torch.cuda.synchronize()
        out.append([i.reshape(width * height, -1) for i in images])
    for images in out[1:]:
        for a, b in zip(out[0], images):
            assert np.count_nonzero((a != b).any(-1)) <= width * height // 20_000
    assert deep.check_errors() == (0, 0)
