"""Batches on either side of the sizes from which a ray has a lane of its own. The sizes go with the nodes that a random
line meets (the last word but one of the kernels' parameters), so each scene has its own; every result must be the
reference order's, except where a ray meets two triangles at exactly the same distance."""

import ctypes as C

import numpy as np
import pytest

from helpers import rt, scenes
from rendiation_gb300 import native
from test_instanced_walks_gpu import grid_scene, params_tail

pytestmark = pytest.mark.gpu


def system(kind, size):
    if kind == "grid":
        return grid_scene(2, size)[1]
    m = scenes.triangle_soup(size, seed=3, offset=0.3) if kind == "soup" else scenes.heightfield(size, seed=4)
    P = rt.AccelerationStructureSystem(device=0)
    b = P.create_bottom_level_acceleration_structure([rt.BottomLevelAccelerationStructureBuildSource(m.positions, m.indices)])
    P.bind_tlas([P.create_top_level_acceleration_structure([rt.TopLevelAccelerationStructureSourceInstance(b)])])
    P.build(blas_bin_size=4, device_build=True)
    return P


def limit(P, per_square, least, most):
    return int(min(max(per_square * params_tail(P)[2] ** 2, least), most))


def camera(kind, width, height):
    return scenes.heightfield_camera(width, height) if kind == "field" else scenes.soup_camera(width, height)


def rays_of(kind, n, seed):
    """Stretches of 96 camera rays and of 96 rays in random directions."""
    cam = scenes.pinhole_rays(camera(kind, 640, -(-n // 640)))[:n]
    lo, hi = ((0, 0, -0.1), (1, 1, 0.4)) if kind == "field" else ((-0.02,) * 3, (1.02,) * 3)
    return np.where(((np.arange(n) + 16) // 96) % 2 == 0, cam, scenes.sphere_rays(n, lo, hi, seed=seed))


SCENES = [("soup", 12), ("soup", 200), ("field", 16), ("field", 64), ("grid", 9), ("grid", 300)]


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("kind,size", SCENES)
def test_queries(cuda, kind, size, watertight):
    import torch

    P = system(kind, size)
    at = limit(P, 300.0, 40_000, 400_000)
    for n in (at - 2, at + 2, at + 33):
        d = torch.from_numpy(rays_of(kind, n, n).view(np.float32).reshape(-1, 8).copy()).cuda()
        out = []
        for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
            hits = torch.full((n, 4), -7.0, device="cuda")
            ext = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
            P.trace(d, hits, ext, traversal=traversal | watertight, local_stack=1 if traversal else 0)
            out.append(np.concatenate([hits.cpu().numpy().view(np.int32), ext.cpu().numpy()], 1))
        for got in out[1:]:
            differ = (got != out[0]).any(1)
            assert np.count_nonzero(differ) <= n // 20_000
            assert np.array_equal(got[differ, 0], out[0][differ, 0])  # the same distance
        assert (out[0][:, 3] != -1).any()
    assert P.check_errors() == (0, 0)


@pytest.mark.parametrize("kind,size", SCENES)
def test_hit_queries(cuda, kind, size):
    import torch

    P = system(kind, size)
    at = limit(P, 255.0, 48_000, 400_000)
    attr = torch.rand(3 * 10_000, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    for n in (at - 2, at + 33):
        d = torch.from_numpy(rays_of(kind, n, n).view(np.float32).reshape(-1, 8).copy()).cuda()
        out = []
        for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
            z = lambda *s, dtype=torch.float32: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
            tri, inst, hit, loss = z(n, dtype=torch.int32), z(n, dtype=torch.int32), z(n, 4), z(1, dtype=torch.float64)
            f = native.HitDiffDesc(rays=d.data_ptr(), count=n, attributes=attr.data_ptr(), traversal=traversal,
                                   hit=hit.data_ptr(), hit_tri=tri.data_ptr(), hit_inst=inst.data_ptr())
            g = native.AttrLossDesc(rays=d.data_ptr(), count=n, attributes=attr.data_ptr(), traversal=traversal,
                                    grad_scale=1.0, loss_sum=loss.data_ptr())
            assert native.lib().rdn_hit_diff_forward(P._h, C.byref(f), None) == 0
            assert native.lib().rdn_attr_loss_forward(P._h, C.byref(g), None) == 0
            torch.cuda.synchronize()
            out.append([t.cpu().numpy() for t in (tri, inst, hit, loss)])
        (tri0, inst0, hit0, loss0), (tri1, inst1, hit1, loss1) = out
        same = (tri0 == tri1) & (inst0 == inst1)
        assert np.count_nonzero(~same) <= n // 20_000 and np.array_equal(hit0[same], hit1[same])
        # a sum of n non-negative doubles in another order, and the ties' own terms (values below 1: at most 1 each)
        assert abs(loss0[0] - loss1[0]) <= 4 * n * 2.0**-53 * loss0[0] + np.count_nonzero(~same)


@pytest.mark.parametrize("kind,size", SCENES)
def test_attribute_paths(cuda, kind, size):
    import torch

    P = system(kind, size)
    at = limit(P, 120.0, 20_000, 150_000)
    attr = torch.rand(3 * 10_000, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    for n in (at - 1, at + 2):
        d = torch.from_numpy(rays_of(kind, n, n).view(np.float32).reshape(-1, 8).copy()).cuda()
        out = []
        for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
            z = lambda *s, dtype=torch.float32: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
            tri, rays, values = z(n, 2, dtype=torch.int32), z(n, 16), z(n, 2)
            f = native.AttrPathDesc(rays=d.data_ptr(), count=n, segments=2, seed=3, attributes=attr.data_ptr(),
                                    grad_scale=1.0, traversal=traversal, seg_tri=tri.data_ptr(),
                                    seg_rays=rays.data_ptr(), values=values.data_ptr())
            assert native.lib().rdn_attr_paths_forward(P._h, C.byref(f), None) == 0
            torch.cuda.synchronize()
            out.append([t.cpu().numpy() for t in (tri, rays, values)])
        same = (out[0][0] == out[1][0]).all(1)
        assert np.count_nonzero(~same) <= n // 20_000
        assert all(np.array_equal(a[same], b[same]) for a, b in zip(*out))


def sides(P, per_square, least, most):
    """Frames (width a multiple of 8, so that tiles have no rest) just below and just above the limit."""
    at = limit(P, per_square, least, most)
    width = max(8, int(at**0.5) // 8 * 8)
    rows = max(1, at // width // 8 * 8)
    return [(width, rows), (width, rows + 8)]


@pytest.mark.parametrize("kind,size", SCENES)
def test_wavefront_frames(cuda, kind, size):
    import torch

    P = system(kind, size)
    frames = sides(P, 155.0, 30_000, 300_000) + [(440, 300), (548, 548)]
    for width, height in frames:
        out = []
        for traversal, phases in ((rt.TRAVERSAL_REFERENCE, (0,)), (rt.TRAVERSAL_ORDERED, (0,)),
                                  (rt.TRAVERSAL_ORDERED_WIDE, (1, 2))):
            wf = rt.Wavefront(P, camera(kind, width, height), (0.2, 0.2, 2.0))
            wf.configure((traversal, 64, 1), (traversal, 64, 1))
            for ph in phases:
                wf.run(5, phases=ph)
            torch.cuda.synchronize()
            out.append((wf.results().copy().view(np.uint32).reshape(-1, 8), wf.rays_traced()))
        for got, rays in out[1:]:
            assert np.count_nonzero((got != out[0][0]).any(-1)) <= width * height // 20_000
            assert rays == out[0][1] and rays[0] == width * height
    assert P.check_errors() == (0, 0)


@pytest.mark.parametrize("kind,size", SCENES)
def test_rendered_frames(cuda, kind, size):
    import torch

    from rendiation_gb300 import path_tracing as pt
    from rendiation_gb300 import task_graph as tg

    P = system(kind, size)
    eye, target = ((0.5, -0.4, 0.6), (0.5, 0.5, 0.0)) if kind == "field" else ((0.5, -1.2, 1.1), (0.5, 0.5, 0.5))
    lights = [pt.directional_light((3.0, 2.5, 2.0), (0.3, 0.2, -1.0))]
    for ao, frames in ((True, sides(P, 180.0, 40_000, 200_000)), (False, sides(P, 90.0, 0, 200_000))):
        for width, height in frames:
            vp = tg.look_at_view_projection_inv(eye, target, (0, 0, 1), 40.0, width / height)
            out = []
            for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
                if ao:
                    R = tg.AmbientOcclusion(P, width, height, vp, eye, traversal=traversal)
                else:
                    R = pt.DeviceReferencePathTracingRenderer(P, width, height, vp, eye, lights=lights,
                                                              traversal=traversal, background_color=(0.3, 0.4, 0.6))
                R.render()
                torch.cuda.synchronize()
                out.append(R.result().copy())
            assert np.count_nonzero((out[0] != out[1]).any(-1)) <= width * height // 20_000
    assert P.check_errors() == (0, 0)


@pytest.mark.parametrize("kind,size", SCENES)
@pytest.mark.parametrize("watertight,sort_key,graph", [(0, 0, True), (rt.INTERSECT_WATERTIGHT, 0, False), (0, 1, False)])
def test_paths(cuda, kind, size, watertight, sort_key, graph):
    import torch

    P = system(kind, size)
    at = limit(P, 260.0, 100_000, 400_000)
    for n in (at - 2, at + 33):
        d = torch.from_numpy(rays_of(kind, n, n).view(np.float32).reshape(-1, 8).copy()).cuda()
        out = []
        for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
            p = rt.Paths(P, d, max_bounces=3, seed=7, traversal=traversal | watertight, sort_key=sort_key)
            if graph:
                p.capture()
                p.launch_graph()
                p.launch_graph()
            else:
                p.run()
            torch.cuda.synchronize()
            out.append((p.results().copy(), p.segments()))
        for got, segments in out[1:]:
            assert np.count_nonzero(got != out[0][0]) <= n // 20_000
            assert all(abs(a - b) <= n // 20_000 for a, b in zip(segments, out[0][1]))
        assert out[0][1][0] == n and out[0][1][1] > 0
    assert P.check_errors() == (0, 0)


def test_paths_of_many_scenes(cuda):
    """Groups that are alike end where the scene changes; an index that is not bound ends its path."""
    import torch

    from test_quads_gpu import soup_system

    P = soup_system([scenes.triangle_soup(k, seed=k, offset=0.05) for k in (300, 2000, 6000)])
    n = limit(P, 260.0, 100_000, 400_000) + 5
    d = torch.from_numpy(rays_of("soup", n, 3).view(np.float32).reshape(-1, 8).copy()).cuda()
    rng = np.random.default_rng(3)
    for tidx in (np.repeat(rng.integers(0, 4, n // 48 + 1), 48)[:n], rng.integers(0, 3, n), np.sort(rng.integers(0, 4, n))):
        t = torch.from_numpy(tidx.astype(np.int32)).cuda()
        out = []
        for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED):
            p = rt.Paths(P, d, t, max_bounces=2, seed=5, traversal=traversal)
            p.run()
            torch.cuda.synchronize()
            out.append(p.results().copy())
        assert np.count_nonzero(out[0] != out[1]) <= n // 20_000
