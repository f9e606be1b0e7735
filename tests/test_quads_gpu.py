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
