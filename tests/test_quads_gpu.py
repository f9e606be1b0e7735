"""Ordered batch queries at the sizes and shapes where their walks change.

The ordered traversals of rdn_trace share a warp out to eight groups of four
lanes or keep one ray per lane, by the ray count and by whether 32 consecutive
rays are alike. Every result must be the reference order's (itself
bit-identical to the oracle, tests/test_trace_gpu.py), except where two
triangles are at exactly the same distance: no other tolerance.
"""

import numpy as np
import pytest

from rendiation_gb300 import raytracing as rt
from rendiation_gb300 import scenes

pytestmark = pytest.mark.gpu


def mixed_rays(n, seed):
    """Stretches of 96 pinhole rays and of 96 rays in random directions, so
    that groups of 32 of both kinds (and, at the seams, of neither) occur."""
    cam = scenes.pinhole_rays(scenes.soup_camera(512, -(-n // 512)))[:n]
    rnd = scenes.sphere_rays(n, (-0.02,) * 3, (1.02,) * 3, seed=seed)
    pick = ((np.arange(n) + 16) // 96) % 2 == 0
    return np.where(pick, cam, rnd)


def check(P, rays, tidx=None, **kw):
    import torch

    d = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    t = None if tidx is None else torch.from_numpy(tidx.astype(np.int32)).cuda()
    n = rays.shape[0]

    def run(traversal):
        hits = torch.full((n, 4), -7.0, device="cuda")
        ext = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
        P.trace(d, hits, ext, tlas_idx=t, traversal=traversal, **kw)
        assert P.check_errors() in ((0, 0), (0, 2))
        return rt.hits_to_numpy(hits), ext.cpu().numpy()

    want, want_ext = run(rt.TRAVERSAL_REFERENCE)
    for traversal in (rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        got, ext = run(traversal)
        same = (got["prim"] == want["prim"]) & (ext == want_ext).all(1)
        for k in ("t", "u", "v"):
            same &= got[k].view(np.uint32) == want[k].view(np.uint32)
        tie = got["t"].view(np.uint32) == want["t"].view(np.uint32)
        assert np.all(same | tie), (traversal, np.flatnonzero(~(same | tie))[:5])
        assert np.count_nonzero(~same) <= 1 + n // 1000
    return want


def soup_system(meshes, **build):
    P = rt.AccelerationStructureSystem(device=0)
    handles = []
    for m in meshes:
        b = P.create_bottom_level_acceleration_structure([rt.BottomLevelAccelerationStructureBuildSource(m.positions)])
        handles.append(P.create_top_level_acceleration_structure([rt.TopLevelAccelerationStructureSourceInstance(b)]))
    P.bind_tlas(handles)
    P.build(**dict(dict(blas_bin_size=4, device_build=True), **build))
    return P


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 33, 39_999, 40_000, 40_033, 99_999, 100_001, 599_999, 600_001])
def test_counts_at_the_edges(cuda, n):
    P = soup_system([scenes.triangle_soup(3000, seed=3)])
    want = check(P, mixed_rays(n, seed=n))
    assert n < 100 or (want["prim"] != rt.MISS).any()


@pytest.mark.parametrize("bin_size,depth,device_build", [(1, 50, True), (7, 50, True), (8, 50, False), (4, 2, True),
                                                         (300, 50, False)])
def test_leaf_sizes(cuda, bin_size, depth, device_build):
    """Leaves of one, seven, eight and hundreds of triangles, and a tree that is a single leaf."""
    P = soup_system([scenes.triangle_soup(n, seed=n) for n in (1, 5, 290, 2000)], blas_bin_size=bin_size,
                    blas_max_depth=depth, device_build=device_build)
    rays = mixed_rays(4096, seed=5)
    tidx = np.random.default_rng(1).integers(0, 5, 4096)  # index 4 is not bound: a miss
    check(P, rays, tidx)
    check(P, rays, np.repeat(np.arange(4), 1024))


@pytest.mark.parametrize("anyhit", [rt.ANYHIT_ACCEPT, rt.ANYHIT_ACCEPT_EVEN_PRIMS, rt.ANYHIT_PRIMITIVE_MASK])
@pytest.mark.parametrize("n", [2000, 60_000])
def test_instances_flags_and_policies(cuda, anyhit, n):
    """Several geometries and overlapping instances per ray, non-opaque triangles, culling, the watertight test."""
    import torch

    src = rt.BottomLevelAccelerationStructureBuildSource
    P = rt.AccelerationStructureSystem(device=0)
    a, b = scenes.triangle_soup(301, seed=1), scenes.triangle_soup(700, seed=2)
    both = P.create_bottom_level_acceleration_structure([src(a.positions, flags=0), src(b.positions, flags=1)])
    one = P.create_bottom_level_acceleration_structure([src(b.positions, flags=0)])
    inst = []
    for k in range(6):
        m = np.eye(4, dtype=np.float32)
        m[:3, :3] *= 0.5 + 0.2 * k
        m[3, :3] = (0.1 * k, -0.05 * k, 0.02 * k)  # columns in memory: translation at 12..14
        inst.append(rt.TopLevelAccelerationStructureSourceInstance((both, one)[k % 2], m.reshape(-1), k,
                                                                   flags=(0, 1, 2)[k % 3]))
    P.bind_tlas([P.create_top_level_acceleration_structure(inst)])
    P.build(blas_bin_size=4)
    words = np.random.default_rng(2).integers(0, 2**31, (1001 + 700 + 63) // 32, dtype=np.int32)
    mask = torch.from_numpy(words).cuda() if anyhit == rt.ANYHIT_PRIMITIVE_MASK else None
    rays = mixed_rays(n, seed=8)
    for flags in (0, rt.RAY_FLAG_CULL_BACK_FACING_TRIANGLES, rt.RAY_FLAG_FORCE_NON_OPAQUE):
        check(P, rays, anyhit_mode=anyhit, anyhit_mask=mask, ray_flags=flags)


@pytest.mark.parametrize("n", [500, 50_000])
def test_first_hit_queries_agree_on_hit_and_miss(cuda, n):
    import torch

    P = soup_system([scenes.triangle_soup(5000, seed=6)])
    d = torch.from_numpy(mixed_rays(n, seed=9).view(np.float32).reshape(-1, 8).copy()).cuda()
    res = {}
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        for kw in (dict(ray_flags=rt.RAY_FLAG_ACCEPT_FIRST_HIT_AND_END_SEARCH),
                   dict(ray_flags=rt.RAY_FLAG_FORCE_NON_OPAQUE, anyhit_mode=rt.ANYHIT_ACCEPT_AND_END)):
            hits = torch.zeros((n, 4), device="cuda")
            P.trace(d, hits, traversal=traversal, **kw)
            res[traversal, str(kw)] = rt.hits_to_numpy(hits)["prim"] != rt.MISS
    first = next(iter(res.values()))
    assert all(np.array_equal(first, r) for r in res.values())


def field_system(n=64):
    m = scenes.heightfield(n, seed=4)
    P = rt.AccelerationStructureSystem(device=0)
    b = P.create_bottom_level_acceleration_structure([rt.BottomLevelAccelerationStructureBuildSource(m.positions, m.indices)])
    P.bind_tlas([P.create_top_level_acceleration_structure([rt.TopLevelAccelerationStructureSourceInstance(b)])])
    P.build(blas_bin_size=4)
    return P, m


def field_rays(n, seed):
    """Stretches of camera rays and of rays in random directions into the field."""
    w = 640
    cam = scenes.pinhole_rays(scenes.heightfield_camera(w, -(-n // w)))[:n]
    rnd = scenes.sphere_rays(n, (0, 0, -0.1), (1, 1, 0.4), seed=seed)
    return np.where(((np.arange(n) + 16) // 96) % 2 == 0, cam, rnd)


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("n", [1, 33, 47_999, 48_001, 399_999, 400_033])
def test_differentiable_batches(cuda, n, watertight):
    """Loss and hit query, forward and traced adjoint, against the reference order: the same hits and values; vertex
    gradients up to the order of their f32 sums (at most m terms a vertex: m 2^-24 of the norm)."""
    import ctypes as C

    import torch
    from rendiation_gb300 import native

    P, mesh = field_system()
    L = native.lib()
    rays = torch.from_numpy(field_rays(n, n).view(np.float32).reshape(-1, 8).copy()).cuda()
    g = torch.Generator(device="cuda").manual_seed(1)
    attr = torch.rand(mesh.positions.shape[0], generator=g, device="cuda")
    target = torch.rand(n, generator=g, device="cuda")
    grad_hit = torch.randn((n, 4), generator=g, device="cuda")

    def run(traversal, query):
        z = lambda *s, dtype=torch.float32: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
        r = dict(tri=z(n, dtype=torch.int32), inst=z(n, dtype=torch.int32), grad=z(attr.shape[0], 4), go=z(n, 3),
                 gd=z(n, 3), loss=z(1, dtype=torch.float64), value=z(n), hit=z(n, 4))
        base = dict(rays=rays.data_ptr(), count=n, attributes=attr.data_ptr(), traversal=traversal | watertight)
        grads = dict(grad_vertices=r["grad"].data_ptr(), grad_ray_origin=r["go"].data_ptr(),
                     grad_ray_direction=r["gd"].data_ptr())
        rec = dict(hit_tri=r["tri"].data_ptr(), hit_inst=r["inst"].data_ptr())
        if query:
            f = native.HitDiffDesc(**base, **rec, hit=r["hit"].data_ptr())
            a = native.HitDiffDesc(**base, **grads, grad_hit=grad_hit.data_ptr())
            assert L.rdn_hit_diff_forward(P._h, C.byref(f), None) == 0
            assert L.rdn_hit_diff_adjoint(P._h, C.byref(a), None) == 0
        else:
            f = native.AttrLossDesc(**base, **rec, targets=target.data_ptr(), ray_value=r["value"].data_ptr(),
                                    loss_sum=r["loss"].data_ptr(), grad_scale=1.0)
            a = native.AttrLossDesc(**base, **grads, targets=target.data_ptr(), grad_scale=1.0)
            assert L.rdn_attr_loss_forward(P._h, C.byref(f), None) == 0
            assert L.rdn_attr_loss_adjoint(P._h, C.byref(a), None) == 0
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in r.items()}

    for query in (False, True):
        want, got = run(rt.TRAVERSAL_REFERENCE, query), run(rt.TRAVERSAL_ORDERED, query)
        same = want["tri"] == got["tri"]
        assert np.count_nonzero(~same) <= 1 + n // 20_000  # exact-distance ties
        for k in ("inst", "value", "hit", "go", "gd"):
            assert np.array_equal(want[k][same], got[k][same]), k
        if same.all():
            assert abs(want["loss"] - got["loss"]) <= 1e-12 * np.abs(want["loss"])
            hit = want["tri"] != -1
            idx = mesh.indices.reshape(-1, 3)[want["tri"][hit]]
            m = np.bincount(idx.reshape(-1), minlength=1).max() if hit.any() else 0
            diff = np.linalg.norm(want["grad"].astype(np.float64) - got["grad"])
            assert diff <= m * 2.0**-24 * np.linalg.norm(want["grad"].astype(np.float64))


@pytest.mark.parametrize("n", [5, 1000, 39_999, 100_001])
def test_path_batches(cuda, n):
    """Paths of both executors against the reference order (a tie may send a path elsewhere)."""
    import torch

    P = soup_system([scenes.triangle_soup(k, seed=k) for k in (400, 3000, 9000)])
    rays = torch.from_numpy(mixed_rays(n, seed=n).view(np.float32).reshape(-1, 8).copy()).cuda()
    tidx = torch.from_numpy(np.random.default_rng(n).integers(0, 3, n).astype(np.int32)).cuda()
    out = {}
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        for watertight in (0, rt.INTERSECT_WATERTIGHT):
            for sort_key in (0, 2):
                p = rt.Paths(P, rays, tidx, max_bounces=3, seed=7, traversal=traversal | watertight, sort_key=sort_key)
                p.run()
                torch.cuda.synchronize()
                out[traversal, watertight, sort_key] = p.results()
                assert P.check_errors() == (0, 0)
    for (traversal, watertight, sort_key), got in out.items():
        assert np.count_nonzero(got != out[rt.TRAVERSAL_REFERENCE, watertight, 0]) <= n // 20_000


@pytest.mark.parametrize("width,height", [(7, 5), (316, 312), (316, 320), (632, 632), (640, 640)])
def test_frames_of_both_walks(cuda, width, height):
    """AO and path-traced frames on either side of the sizes where their walks change, against the reference order:
    the same texels, except where a ray meets two triangles at exactly the same distance."""
    import torch

    from rendiation_gb300 import path_tracing as pt
    from rendiation_gb300 import task_graph as tg

    P, _ = field_system(128)
    eye = (0.5, -0.4, 0.6)
    vp = tg.look_at_view_projection_inv(eye, (0.5, 0.5, 0.0), (0, 0, 1), 40.0, width / height)
    lights = [pt.directional_light((3.0, 2.5, 2.0), (0.3, 0.2, -1.0))]
    images = {}
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        ao = tg.AmbientOcclusion(P, width, height, vp, eye, traversal=traversal)
        ao.sample_count = 200
        ao.render()
        R = pt.DeviceReferencePathTracingRenderer(P, width, height, vp, eye, lights=lights, traversal=traversal,
                                                  background_color=(0.3, 0.4, 0.6), count_rays=True)
        R.render()
        torch.cuda.synchronize()
        images[traversal] = ao.result().copy(), R.result().copy(), R.rays_traced()
    want = images[rt.TRAVERSAL_REFERENCE]
    n = width * height
    for traversal in (rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        for k in (0, 1):
            assert np.count_nonzero((images[traversal][k] != want[k]).any(-1)) <= n // 20_000
        assert all(abs(a - b) <= 3 * (n // 20_000) for a, b in zip(images[traversal][2], want[2]))
    assert P.check_errors() == (0, 0)


@pytest.mark.parametrize("width,height", [(3, 9), (320, 312), (316, 320), (670, 670), (680, 672)])
def test_wavefront_frames_of_both_walks(cuda, width, height):
    """Wavefront frames on either side of the sizes where their walks change: every record of the reference order's
    frame, except after an exact-distance tie."""
    import torch

    P, _ = field_system(128)
    cam = scenes.heightfield_camera(width, height)
    frames = {}
    for watertight in (0, rt.INTERSECT_WATERTIGHT):
        for traversal, refill, local in ((rt.TRAVERSAL_REFERENCE, 0, 0), (rt.TRAVERSAL_ORDERED, 0, 1),
                                         (rt.TRAVERSAL_ORDERED_WIDE, 0, 0), (rt.TRAVERSAL_ORDERED, 8, 0)):
            wf = rt.Wavefront(P, cam, (0.2, 0.2, 2.0))
            knobs = (traversal | watertight, 64, local)
            wf.configure(knobs, knobs, refill=refill)
            wf.run(3)
            torch.cuda.synchronize()
            frames[watertight, traversal, refill] = wf.results().copy(), wf.rays_traced()
    for (watertight, traversal, refill), (got, rays) in frames.items():
        want, want_rays = frames[watertight, rt.TRAVERSAL_REFERENCE, 0]
        assert np.count_nonzero(got.view(np.uint32).reshape(-1, 8) != want.view(np.uint32).reshape(-1, 8)) <= \
            8 * (width * height // 20_000)
        assert rays == want_rays
    assert P.check_errors() == (0, 0)


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("n", [1, 33, 150_000, 150_001])
def test_attribute_paths_at_the_edges(cuda, n, watertight):
    """Differentiable paths on both sides of the size from which a lane takes a path."""
    import ctypes as C

    import torch

    from rendiation_gb300 import native

    P, mesh = field_system()
    L = native.lib()
    rays = torch.from_numpy(field_rays(n, n).view(np.float32).reshape(-1, 8).copy()).cuda()
    g = torch.Generator(device="cuda").manual_seed(2)
    attr = torch.rand(mesh.positions.shape[0], generator=g, device="cuda")
    target = torch.rand(2 * n, generator=g, device="cuda")

    def run(traversal):
        z = lambda *s, dtype=torch.float32: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
        r = dict(tri=z(n, 2, dtype=torch.int32), inst=z(n, 2, dtype=torch.int32), rays=z(n, 16), values=z(n, 2),
                 loss=z(1, dtype=torch.float64), grad=z(attr.shape[0], 4))
        base = dict(rays=rays.data_ptr(), count=n, segments=2, seed=3, attributes=attr.data_ptr(),
                    targets=target.data_ptr(), grad_scale=1.0, traversal=traversal | watertight)
        f = native.AttrPathDesc(**base, seg_tri=r["tri"].data_ptr(), seg_inst=r["inst"].data_ptr(),
                                seg_rays=r["rays"].data_ptr(), values=r["values"].data_ptr(),
                                loss_sum=r["loss"].data_ptr())
        a = native.AttrPathDesc(**base, grad_vertices=r["grad"].data_ptr())
        assert L.rdn_attr_paths_forward(P._h, C.byref(f), None) == 0
        assert L.rdn_attr_paths_adjoint(P._h, C.byref(a), None) == 0
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in r.items()}

    want, got = run(rt.TRAVERSAL_REFERENCE), run(rt.TRAVERSAL_ORDERED)
    same = (want["tri"] == got["tri"]).all(1)
    assert np.count_nonzero(~same) <= 1 + n // 20_000  # exact-distance ties
    for k in ("inst", "rays", "values"):
        assert np.array_equal(want[k][same], got[k][same]), k
    # a sum of n non-negative doubles in another order, and the ties' own terms (at most 1 each)
    assert abs(want["loss"][0] - got["loss"][0]) <= 4 * n * 2.0**-53 * abs(want["loss"][0]) + 2 * np.count_nonzero(~same)
    if same.all():
        hit = want["tri"] != -1
        m = np.bincount(mesh.indices.reshape(-1, 3)[want["tri"][hit]].reshape(-1), minlength=1).max() if hit.any() else 0
        diff = np.linalg.norm(want["grad"].astype(np.float64) - got["grad"])
        assert diff <= m * 2.0**-24 * np.linalg.norm(want["grad"].astype(np.float64))


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("width,height", [(1, 1), (7, 5), (33, 31), (250, 200)])
def test_task_graph_trace_polls(cuda, width, height, watertight):
    """The AO pipeline on the task graph (its trace tasks start and wait in the same warps) against the reference order."""
    import torch

    from rendiation_gb300 import task_graph as tg

    P, _ = field_system(128)
    eye = (0.5, -0.4, 0.6)
    vp = tg.look_at_view_projection_inv(eye, (0.5, 0.5, 0.0), (0, 0, 1), 40.0, width / height)
    images = []
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED, rt.TRAVERSAL_ORDERED_WIDE):
        ao = tg.AmbientOcclusion(P, width, height, vp, eye, traversal=traversal | watertight, mode="graph")
        ao.sample_count = 200
        ao.render()
        torch.cuda.synchronize()
        images.append(ao.result().copy())
    for image in images[1:]:
        assert np.count_nonzero((image != images[0]).any(-1)) <= width * height // 20_000
    assert P.check_errors() == (0, 0)
