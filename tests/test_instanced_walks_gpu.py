"""Structures of several instances a TLAS: the walks that they are given in frames, paths and the path tracer against
the reference order (the same results, except where a ray meets two triangles at exactly the same distance), and the
measure of a tree by which walks are chosen."""

import ctypes as C
import struct

import numpy as np
import pytest

from helpers import Scene, mat4_cols, rot_x, rot_z, rt, scenes

pytestmark = pytest.mark.gpu


def grid_scene(k, tris, device_build=True):
    """k^3 turned instances of two BLASes (one of two geometries, partly not opaque) next to each other and overlapping."""
    a, b = scenes.triangle_soup(tris, seed=1), scenes.triangle_soup(tris // 2 + 1, seed=2)
    blas = [[(a.positions, None, 1)], [(b.positions, None, 0), (a.positions[: 3 * (tris // 3)], None, 1)]]
    inst = []
    for i in range(k**3):
        at = np.array([i % k, i // k % k, i // k // k]) / k
        inst.append({"blas": 0 if i % 5 else 1, "transform": mat4_cols(rot_z(0.3 * i) @ rot_x(0.1 * i), (1.1 / k,) * 3, at),
                     "custom": i, "mask": 0xFF if i % 7 else 0x3})
    sc = Scene(blas, [inst])
    return sc, sc.build_product(device_build=device_build)


def params_tail(P):
    """(packed, instanced, line_nodes), the last words of the kernels' parameter block."""
    size = C.c_size_t(0)
    assert P._L.rdn_trace_params(P._h, 1, None, C.byref(size)) == 0
    buf = (C.c_uint8 * size.value)()
    assert P._L.rdn_trace_params(P._h, 1, buf, C.byref(size)) == 0
    return struct.unpack_from("<IIf", bytes(buf), size.value - 16)


def line_nodes_of(P):
    """Mean over single-instance TLASes of the binary inner nodes, by their area over the root's, in 64 bits."""
    f = np.frombuffer(P.built_array("tri_bvh_forest"), np.float32).reshape(-1, 12)
    u = f.view(np.uint32)
    roots = np.frombuffer(P.built_array("tri_bvh_root"), np.uint32).reshape(-1, 4)[:, 0]
    d = f[:, 4:7].astype(np.float64) - f[:, 0:3]
    area = d[:, 0] * d[:, 1] + d[:, 0] * d[:, 2] + d[:, 1] * d[:, 2]
    sums = [1.0 + area[s:e][u[s:e, 3] != u[s:e, 7]].sum() / area[s] for s, e in zip(roots, [*roots[1:], len(f)])]
    return np.mean(sums)


@pytest.mark.parametrize("sizes", [[3000], [700, 5, 1, 4000, 60, 300], [17] * 40])
def test_line_nodes(cuda, sizes):
    sc = Scene([[(scenes.triangle_soup(n, seed=k).positions, None, 1)] for k, n in enumerate(sizes)],
               [[{"blas": k}] for k in range(len(sizes))])
    values = []
    for device_build in (False, True, True):
        P = sc.build_product(device_build=device_build)
        packed, instanced, nodes = params_tail(P)
        assert (packed, instanced) == (1, 0)
        values.append(nodes)
    want = line_nodes_of(P)
    assert values[1] == values[2]  # sums of whole numbers: the same from build to build
    # areas in f32 (three roundings of 2^-24 each), a share cut at 2^-24: below 2^-22 a node and 2^-21 of the sum
    assert all(abs(v - want) <= 2.0**-21 * want + 2.0**-22 * max(sizes) for v in values)


def test_instanced_flag(cuda):
    _, P = grid_scene(2, 100)
    assert params_tail(P)[:2] == (1, 1)
    m = scenes.triangle_soup(10, seed=1)
    two = Scene([[(m.positions, None, 1)]], [[{"blas": 0}], [{"blas": 0}, {"blas": 0}], []]).build_product()
    assert params_tail(two)[1] == 1


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("schedule", [0, 1, 2])
@pytest.mark.parametrize("k,tris,width,height", [(3, 3000, 640, 400), (2, 30, 61, 35), (4, 1000, 333, 201)])
def test_path_tracer(cuda, schedule, watertight, k, tris, width, height):
    import torch

    from rendiation_gb300 import path_tracing as pt
    from rendiation_gb300 import task_graph as tg

    _, P = grid_scene(k, tris)
    eye = (0.5, -1.2, 1.1)
    vp = tg.look_at_view_projection_inv(eye, (0.5, 0.5, 0.5), (0, 0, 1), 40.0, width / height)
    lights = [pt.directional_light((3.0, 2.5, 2.0), (0.3, 0.2, -1.0))]
    images = []
    for traversal in (rt.TRAVERSAL_REFERENCE, rt.TRAVERSAL_ORDERED_WIDE):
        R = pt.DeviceReferencePathTracingRenderer(P, width, height, vp, eye, lights=lights, schedule=schedule,
                                                  traversal=traversal | watertight, background_color=(0.3, 0.4, 0.6))
        R.render()
        torch.cuda.synchronize()
        images.append(R.result().copy())
    assert np.count_nonzero((images[0] != images[1]).any(-1)) <= width * height // 20_000
    assert (images[0] != images[0][0]).any() and P.check_errors() == (0, 0)


@pytest.mark.parametrize("watertight", [0, rt.INTERSECT_WATERTIGHT])
@pytest.mark.parametrize("width,height", [(40, 30), (700, 460)])
def test_frames(cuda, width, height, watertight):
    """Secondary rays of instanced structures: also where the primaries have a lane each, and phase by phase."""
    import torch

    _, P = grid_scene(3, 200)
    cam = scenes.soup_camera(width, height)
    frames = []
    for traversal, phases in ((rt.TRAVERSAL_REFERENCE, (0,)), (rt.TRAVERSAL_ORDERED_WIDE, (0,)),
                              (rt.TRAVERSAL_ORDERED, (1, 2)), (rt.TRAVERSAL_ORDERED, (3,))):
        wf = rt.Wavefront(P, cam, (0.2, 0.2, 2.0))
        knobs = (traversal | watertight, 64, 1)
        wf.configure(knobs, knobs)
        for ph in phases:
            wf.run(5, phases=ph)
        torch.cuda.synchronize()
        frames.append((wf.results().copy().view(np.uint32).reshape(-1, 8), wf.rays_traced()))
    for got, rays in frames[1:]:
        assert np.count_nonzero((got != frames[0][0]).any(-1)) <= width * height // 20_000
        assert rays == frames[0][1] and rays[1] > 0
    assert P.check_errors() == (0, 0)


@pytest.mark.parametrize("n", [77, 150_001])
def test_attribute_paths(cuda, n):
    import torch

    from rendiation_gb300 import native

    _, P = grid_scene(3, 200)
    L = native.lib()
    rays = torch.from_numpy(scenes.sphere_rays(n, (0,) * 3, (1,) * 3, seed=n).view(np.float32).reshape(-1, 8).copy()).cuda()
    g = torch.Generator(device="cuda").manual_seed(2)
    attr = torch.rand(3 * 400, generator=g, device="cuda")
    target = torch.rand(2 * n, generator=g, device="cuda")

    def run(traversal):
        z = lambda *s, dtype=torch.float32: torch.zeros(s, dtype=dtype, device="cuda")  # noqa: E731
        r = dict(tri=z(n, 2, dtype=torch.int32), inst=z(n, 2, dtype=torch.int32), rays=z(n, 16), values=z(n, 2))
        d = native.AttrPathDesc(rays=rays.data_ptr(), count=n, segments=2, seed=3, attributes=attr.data_ptr(),
                                targets=target.data_ptr(), grad_scale=1.0, traversal=traversal, seg_tri=r["tri"].data_ptr(),
                                seg_inst=r["inst"].data_ptr(), seg_rays=r["rays"].data_ptr(), values=r["values"].data_ptr())
        assert L.rdn_attr_paths_forward(P._h, C.byref(d), None) == 0
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in r.items()}

    want, got = run(rt.TRAVERSAL_REFERENCE), run(rt.TRAVERSAL_ORDERED)
    same = (want["tri"] == got["tri"]).all(1) & (want["inst"] == got["inst"]).all(1)
    assert np.count_nonzero(~same) <= n // 20_000
    assert all(np.array_equal(want[k][same], got[k][same]) for k in ("rays", "values"))
