"""Performance cases of the ray-query path, measured through its public entry points.

Each case is one call (or the short run of calls) that a program using the
package makes again and again: a batch query, a frame, a bounce loop over many
scenes, one step of a differentiable render, a rebuild, the queue primitives.
``listed`` names the cases, ``draw`` gives more of the same ranges,
``prepare`` makes the scene, the inputs and the plan a program keeps, ``run``
makes one pass and ``work`` says what the pass cannot do without. ``exact``
gives a pass's results in 64 bits where they are single formulas of the inputs.

Scenes are the seeded ones of ``rendiation_gb300.scenes``: triangle soups
(10,000 triangles in the plain configuration, 1k to 200k in the batched one)
and heightfields (64 to 1024 vertices a side).
"""

from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from rendiation_gb300 import native, scenes
from rendiation_gb300 import path_tracing as pt
from rendiation_gb300 import raytracing as rt
from rendiation_gb300 import task_graph as tg

TRAVERSALS = {"ordered": rt.TRAVERSAL_ORDERED, "wide": rt.TRAVERSAL_ORDERED_WIDE,
              "reference": rt.TRAVERSAL_REFERENCE}
LIGHT = (0.2, 0.2, 2.0)


def listed():
    return [
        # A probe: a thousand rays into a small scene (picking, visibility tests of a few objects). All latency.
        dict(name="query_1k", kind="query", mesh="soup", size=10_000, rays="sphere", width=1000, height=1,
             traversal="ordered", watertight=False, context=False, block=0, local=0),
        # The plain closest-hit configuration: 10k soup, 256x256 pinhole rays, the call's default knobs.
        dict(name="query_soup", kind="query", mesh="soup", size=10_000, rays="camera", width=256, height=256,
             traversal="ordered", watertight=False, context=False, block=0, local=0),
        # Incoherent rays (a light probe or a bounce batch of the caller's own), an odd count, the watertight test and
        # the hit context a shader reads.
        dict(name="query_sphere", kind="query", mesh="soup", size=150_000, rays="sphere", width=777_777, height=1,
             traversal="wide", watertight=True, context=True, block=0, local=1),
        # The wavefront configuration: primaries, one bounce and one shadow ray per hit, 1080p, tuned knobs.
        dict(name="frame_1080p", kind="frame", size=1024, width=1920, height=1080, traversal="wide", block=64, local=1,
             speculation=2, watertight=False),
        # Many scenes of uneven size, up to 4 diffuse bounces with roulette, replayed from a captured graph.
        dict(name="paths_64", kind="paths", scenes=64, tris=200_000, rays=262_144, bounces=4, sort=0, traversal="ordered",
             local=1, speculation=4),
        # The differentiable configuration: forward and adjoint of the attribute loss, the adjoint tracing again.
        dict(name="loss_256", kind="loss", size=256, width=512, height=512, record=False, traversal="ordered", local=1,
             speculation=4),
        # The general differentiable query: forward with its record, adjoint of all four outputs from the record.
        dict(name="hit_diff", kind="hit_diff", size=128, width=511, height=389, record=True, traversal="ordered",
             local=1, speculation=0),
        # Batched differentiable paths: heightfields of uneven size, 2 bounces, forward + adjoint in one graph.
        dict(name="path_loss_16", kind="path_loss", scenes=16, size=512, rays=400_000, segments=3, record=False,
             traversal="ordered", local=1, speculation=4),
        # Ambient occlusion at the reference's render size, 4 of a still camera's 256 samples, fused kernel.
        dict(name="ao_512", kind="ao", size=1024, width=512, height=512, samples=4, mode="fused", traversal="wide"),
        # The path tracer at the reference's render size for a 1080p frame, the renderer's defaults.
        dict(name="path_trace", kind="path_trace", size=1024, width=682, height=384, samples=2, depth=3, schedule=1,
             lights=1, traversal="wide"),
        # A rebuild on the device (geometry changed), then a first query on the new tree.
        dict(name="rebuild_2m", kind="rebuild", mesh="field", size=1024, rays="camera", width=320, height=180),
        # The queue primitives on a queue of the caller's: a pair sort, a compaction and a scan of an odd count.
        dict(name="regroup_4m", kind="regroup", count=4_000_003, key_bits=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "frame", "paths", "loss", "hit_diff", "path_loss", "ao", "path_trace", "rebuild",
                       "regroup"])
    wide = rng.choice(["ordered", "wide"])
    if kind == "query":
        mesh = rng.choice(["soup", "field"])
        size = _log(rng, 1000, 200_000) if mesh == "soup" else _log(rng, 64, 1024)
        if rng.random() < 0.5:
            w, h = _log(rng, 16, 1920), _log(rng, 16, 1080)
            return dict(kind=kind, mesh=mesh, size=size, rays="camera", width=w, height=h, traversal=wide,
                        watertight=rng.random() < 0.25, context=rng.random() < 0.5, block=rng.choice([0, 64, 128]),
                        local=rng.choice([0, 1]))
        return dict(kind=kind, mesh=mesh, size=size, rays="sphere", width=_log(rng, 100, 1_000_000), height=1,
                    traversal=wide, watertight=rng.random() < 0.25, context=rng.random() < 0.5,
                    block=rng.choice([0, 32, 128]), local=rng.choice([0, 1]))
    if kind == "frame":
        return dict(kind=kind, size=_log(rng, 64, 1024), width=_log(rng, 64, 1920), height=_log(rng, 64, 1080),
                    traversal=wide, block=rng.choice([0, 32, 64, 128]), local=rng.choice([0, 1]),
                    speculation=rng.choice([0, 2, 4]), watertight=rng.random() < 0.25)
    if kind == "paths":
        return dict(kind=kind, scenes=_log(rng, 1, 64), tris=_log(rng, 4000, 200_000), rays=_log(rng, 8192, 262_144),
                    bounces=rng.randint(1, 4), sort=rng.choice([0, 0, 1, 2]), traversal=wide, local=rng.choice([0, 1]),
                    speculation=rng.choice([0, 4]))
    if kind == "loss":
        return dict(kind=kind, size=_log(rng, 64, 256), width=_log(rng, 64, 512), height=_log(rng, 64, 512),
                    record=rng.random() < 0.5, traversal=wide, local=rng.choice([0, 1]), speculation=rng.choice([0, 4]))
    if kind == "hit_diff":
        return dict(kind=kind, size=_log(rng, 32, 256), width=_log(rng, 64, 512), height=_log(rng, 64, 512),
                    record=rng.random() < 0.5, traversal=wide, local=rng.choice([0, 1]), speculation=rng.choice([0, 4]))
    if kind == "path_loss":
        return dict(kind=kind, scenes=_log(rng, 2, 16), size=_log(rng, 96, 512), rays=_log(rng, 64_000, 400_000),
                    segments=rng.randint(2, 3), record=rng.random() < 0.5, traversal=wide, local=1,
                    speculation=rng.choice([0, 4]))
    if kind == "ao":
        return dict(kind=kind, size=_log(rng, 64, 1024), width=_log(rng, 64, 512), height=_log(rng, 64, 512),
                    samples=rng.randint(1, 4), mode=rng.choice(["fused", "graph"]), traversal=wide)
    if kind == "path_trace":
        return dict(kind=kind, size=_log(rng, 64, 1024), width=_log(rng, 64, 682), height=_log(rng, 64, 384),
                    samples=rng.randint(1, 2), depth=rng.randint(1, 3), schedule=rng.choice([0, 1, 1, 2]),
                    lights=rng.randint(0, 2), traversal=wide)
    if kind == "rebuild":
        mesh = rng.choice(["soup", "field"])
        return dict(kind=kind, mesh=mesh, size=_log(rng, 1000, 200_000) if mesh == "soup" else _log(rng, 64, 1024),
                    rays="camera", width=_log(rng, 64, 512), height=_log(rng, 64, 256))
    # the queue primitives on a bounce queue of the caller's: sort by key, compact, scan
    return dict(kind="regroup", count=_log(rng, 1000, 8_000_000), key_bits=rng.choice([8, 16, 24, 32]))


# ---- scenes and inputs ---------------------------------------------------------------------------------------------

def _mesh(case, seed):
    if case["mesh"] == "soup":
        return scenes.triangle_soup(case["size"], seed=seed)
    return scenes.heightfield(case["size"], seed=seed)


def _system(meshes, device_build=True):
    P = rt.AccelerationStructureSystem(device=0)
    handles = []
    for m in meshes:
        b = P.create_bottom_level_acceleration_structure(
            [rt.BottomLevelAccelerationStructureBuildSource(m.positions, m.indices)])
        handles.append(P.create_top_level_acceleration_structure([rt.TopLevelAccelerationStructureSourceInstance(b)]))
    P.bind_tlas(handles)
    P.build(blas_bin_size=4, device_build=device_build)
    return P


def _cuda_rays(rays):
    return torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()


def _camera(mesh_kind, width, height, seed):
    """The workloads' cameras, the field's moved a little by the seed (a camera on the move)."""
    if mesh_kind == "soup":
        return scenes.soup_camera(width, height)
    r = np.random.Generator(np.random.PCG64(seed))
    eye = np.array([0.5, -0.5, 0.8]) + r.uniform(-0.02, 0.02, 3)
    return scenes.PinholeCamera.look_at(eye, (0.5, 0.5, 0.0), 20.0, width, height)


def _rays(case, seed):
    if case["rays"] == "sphere":
        lo, hi = ((-0.02,) * 3, (1.02,) * 3) if case["mesh"] == "soup" else ((0, 0, -0.1), (1, 1, 0.4))
        return scenes.sphere_rays(case["width"] * case["height"], lo, hi, seed=seed + 1)
    return scenes.pinhole_rays(_camera(case["mesh"], case["width"], case["height"], seed))


def _traversal(case):
    return TRAVERSALS[case["traversal"]] | (rt.INTERSECT_WATERTIGHT if case.get("watertight") else 0)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ok(status):
    if status != native.RDN_OK:
        raise native.RdnError(status, "call failed")


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


# ---- batch query ---------------------------------------------------------------------------------------------------

def _prepare_query(case, seed):
    P = _system([_mesh(case, seed)])
    rays = _cuda_rays(_rays(case, seed))
    n = rays.shape[0]
    return dict(kind="query", P=P, rays=rays, hits=torch.zeros((n, 4), device="cuda"),
                ext=torch.zeros((n, 4), dtype=torch.int32, device="cuda") if case["context"] else None,
                knobs=dict(traversal=_traversal(case), block_size=case["block"], local_stack=case["local"]))


def _hit_outputs(hits, ext=None):
    """The hit records by column: distance and barycentrics as numbers, the primitive as a whole number."""
    out = dict(tuv=hits[:, :3], prim=hits.view(torch.int32)[:, 3])
    if ext is not None:
        out["context"] = ext
    return out


def _run_query(s):
    s["P"].trace(s["rays"], s["hits"], s["ext"], **s["knobs"])
    return _hit_outputs(s["hits"], s["ext"])


# ---- wavefront frame -----------------------------------------------------------------------------------------------

def _prepare_frame(case, seed):
    P = _system([scenes.heightfield(case["size"], seed=seed)])
    wf = rt.Wavefront(P, _camera("field", case["width"], case["height"], seed), LIGHT)
    knobs = (_traversal(case), case["block"], case["local"], 0, case["speculation"])
    wf.configure(knobs, knobs)
    return dict(kind="frame", P=P, wf=wf, sample=seed % 1000)


def _run_frame(s):
    wf = s["wf"]
    wf.run(s["sample"])
    words, numbers = wf.out, wf.out.view(torch.float32)
    # rdn_pixel_result: primary prim, t, bounce prim, t, flags, light, direct, instance
    return dict(prims=words[:, 0:3:2], distances=numbers[:, 1:4:2], flags=words[:, 4:6], direct=numbers[:, 6],
                instance=words[:, 7], rays=wf.ray_counts)


# ---- many scenes, diffuse paths ------------------------------------------------------------------------------------

def _paths_sizes(case):
    return (scenes.log_uniform_ints(case["scenes"], 1000, case["tris"], 2),
            scenes.log_uniform_ints(case["scenes"], 4096, case["rays"], 3))


def _prepare_paths(case, seed):
    tris, counts = _paths_sizes(case)
    P = _system([scenes.triangle_soup(int(t), seed=seed + k) for k, t in enumerate(tris)])
    rays = _cuda_rays(scenes.sphere_rays(int(sum(counts)), (-0.02,) * 3, (1.02,) * 3, seed=seed + 50_000))
    tidx = torch.from_numpy(np.repeat(np.arange(len(counts), dtype=np.int32), counts)).cuda()
    paths = rt.Paths(P, rays, tidx, max_bounces=case["bounces"], rr_start=2, seed=seed & 0xFFFF,
                     traversal=_traversal(case), sort_key=case["sort"])
    paths.configure(local_stack=case["local"], speculation=case["speculation"])
    paths.capture()
    return dict(kind="paths", P=P, paths=paths)


def _run_paths(s):
    p = s["paths"]
    p.launch_graph()
    return dict(radiance=p.out[:, 0], depth_flags=p.out.view(torch.int32)[:, 1], segments=p.segments_dev)


# ---- differentiable forms ------------------------------------------------------------------------------------------

def _field_and_target(case, seed):
    mesh = scenes.heightfield(case["size"], seed=seed)
    r = np.random.Generator(np.random.PCG64(seed + 17))
    attr = torch.from_numpy(r.random(mesh.positions.shape[0]).astype(np.float32)).cuda()
    rays = _cuda_rays(scenes.pinhole_rays(_camera("field", case["width"], case["height"], seed)))
    return mesh, attr, rays, torch.from_numpy(r.random(rays.shape[0]).astype(np.float32)).cuda()


def _prepare_loss(case, seed):
    mesh, attr, rays, target = _field_and_target(case, seed)
    P, n = _system([mesh]), rays.shape[0]
    s = dict(kind="loss", P=P, attr=attr, rays=rays, target=target, loss=torch.zeros(1, dtype=torch.float64, device="cuda"),
             value=torch.zeros(n, device="cuda"), grad=torch.zeros((attr.shape[0], 4), device="cuda"),
             grad_o=torch.zeros((n, 3), device="cuda"), grad_d=torch.zeros((n, 3), device="cuda"),
             tri=torch.zeros(n, dtype=torch.int32, device="cuda"), inst=torch.zeros(n, dtype=torch.int32, device="cuda"))
    base = dict(rays=rays.data_ptr(), count=n, attributes=attr.data_ptr(), targets=target.data_ptr(), grad_scale=1.0,
                traversal=_traversal(case), local_stack=case["local"], speculation=case["speculation"],
                hit_tri=s["tri"].data_ptr(), hit_inst=s["inst"].data_ptr())
    s["fwd"] = native.AttrLossDesc(**base, ray_value=s["value"].data_ptr(), loss_sum=s["loss"].data_ptr())
    s["adj"] = native.AttrLossDesc(**base, grad_vertices=s["grad"].data_ptr(), grad_ray_origin=s["grad_o"].data_ptr(),
                                   grad_ray_direction=s["grad_d"].data_ptr(), from_record=int(case["record"]))
    return s


def _run_loss(s):
    L, st = native.lib(), _stream()
    s["loss"].zero_()
    s["grad"].zero_()
    _ok(L.rdn_attr_loss_forward(s["P"]._h, C.byref(s["fwd"]), st))
    _ok(L.rdn_attr_loss_adjoint(s["P"]._h, C.byref(s["adj"]), st))
    return dict(loss=s["loss"], value=s["value"], tri=s["tri"], grad=s["grad"], grad_origin=s["grad_o"],
                grad_direction=s["grad_d"])


def _prepare_hit_diff(case, seed):
    mesh, attr, rays, _ = _field_and_target(case, seed)
    P, n = _system([mesh]), rays.shape[0]
    r = np.random.Generator(np.random.PCG64(seed + 29))
    s = dict(kind="hit_diff", P=P, attr=attr, rays=rays, hit=torch.zeros((n, 4), device="cuda"),
             grad_hit=torch.from_numpy(r.normal(size=(n, 4)).astype(np.float32)).cuda(),
             grad=torch.zeros((attr.shape[0], 4), device="cuda"), grad_o=torch.zeros((n, 3), device="cuda"),
             grad_d=torch.zeros((n, 3), device="cuda"), tri=torch.zeros(n, dtype=torch.int32, device="cuda"),
             inst=torch.zeros(n, dtype=torch.int32, device="cuda"))
    base = dict(rays=rays.data_ptr(), count=n, attributes=attr.data_ptr(), traversal=_traversal(case),
                local_stack=case["local"], speculation=case["speculation"], hit_tri=s["tri"].data_ptr(),
                hit_inst=s["inst"].data_ptr())
    s["fwd"] = native.HitDiffDesc(**base, hit=s["hit"].data_ptr())
    s["adj"] = native.HitDiffDesc(**base, grad_hit=s["grad_hit"].data_ptr(), grad_vertices=s["grad"].data_ptr(),
                                  grad_ray_origin=s["grad_o"].data_ptr(), grad_ray_direction=s["grad_d"].data_ptr(),
                                  from_record=int(case["record"]))
    return s


def _run_hit_diff(s):
    L, st = native.lib(), _stream()
    s["grad"].zero_()
    _ok(L.rdn_hit_diff_forward(s["P"]._h, C.byref(s["fwd"]), st))
    _ok(L.rdn_hit_diff_adjoint(s["P"]._h, C.byref(s["adj"]), st))
    return dict(hit=s["hit"], tri=s["tri"], grad=s["grad"], grad_origin=s["grad_o"], grad_direction=s["grad_d"])


def _path_loss_sizes(case):
    grids = np.sqrt(scenes.log_uniform_ints(case["scenes"], 64 * 64, case["size"] ** 2, 31)).astype(np.int64)
    return grids, scenes.log_uniform_ints(case["scenes"], 32_000, case["rays"], 32)


def _prepare_path_loss(case, seed):
    grids, counts = _path_loss_sizes(case)
    meshes = [scenes.heightfield(int(g), seed=seed + k) for k, g in enumerate(grids)]
    P = _system(meshes)
    rays, tidx = [], []
    for k, c in enumerate(counts):
        w = int(math.sqrt(c * 16 / 9))
        rays.append(scenes.pinhole_rays(_camera("field", w, max(1, int(c) // w), seed + k)))
        tidx.append(np.full(rays[-1].shape[0], k, np.int32))
    rays, tidx = _cuda_rays(np.concatenate(rays)), torch.from_numpy(np.concatenate(tidx)).cuda()
    n, seg, nv = rays.shape[0], case["segments"], sum(m.positions.shape[0] for m in meshes)
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(kind="path_loss", P=P, rays=rays, tidx=tidx, attr=torch.rand(nv, generator=g, device="cuda"),
             targets=torch.rand(n * seg, generator=g, device="cuda"), values=torch.zeros(n * seg, device="cuda"),
             loss=torch.zeros(1, dtype=torch.float64, device="cuda"), grad=torch.zeros((nv, 4), device="cuda"))
    d = native.AttrPathDesc(rays=rays.data_ptr(), tlas_idx=tidx.data_ptr(), count=n, segments=seg, seed=seed & 0xFFFF,
                            attributes=s["attr"].data_ptr(), targets=s["targets"].data_ptr(),
                            values=s["values"].data_ptr(), loss_sum=s["loss"].data_ptr(),
                            grad_vertices=s["grad"].data_ptr(), grad_scale=1.0, traversal=_traversal(case),
                            local_stack=case["local"], speculation=case["speculation"])
    if case["record"]:
        s["tape"] = [torch.zeros(n * seg, dtype=torch.int32, device="cuda"),
                     torch.zeros(n * seg, dtype=torch.int32, device="cuda"), torch.zeros((n * seg, 8), device="cuda")]
        d.seg_tri, d.seg_inst, d.seg_rays = (t.data_ptr() for t in s["tape"])
        d.from_record = 1
    h = C.c_void_p()
    _ok(native.lib().rdn_attr_paths_graph(P._h, C.byref(d), nv, C.byref(h)))
    s["graph"] = _Graph(h)
    return s


class _Graph:
    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        native.lib().rdn_graph_destroy(self.handle)


def _run_path_loss(s):
    _ok(native.lib().rdn_graph_launch(s["graph"].handle, _stream()))
    return dict(loss=s["loss"], values=s["values"], grad=s["grad"])


# ---- renderers -----------------------------------------------------------------------------------------------------

def _view(case, seed, eye, fov):
    r = np.random.Generator(np.random.PCG64(seed))
    eye = tuple(np.asarray(eye) + r.uniform(-0.02, 0.02, 3))
    return tg.look_at_view_projection_inv(eye, (0.5, 0.5, 0.0), (0, 0, 1), fov, case["width"] / case["height"]), eye


def _prepare_ao(case, seed):
    P = _system([scenes.heightfield(case["size"], seed=seed)])
    vp, eye = _view(case, seed, (0.5, -0.5, 0.8), 20.0)
    ao = tg.AmbientOcclusion(P, case["width"], case["height"], vp, eye, traversal=_traversal(case), mode=case["mode"])
    return dict(kind="ao", P=P, ao=ao, samples=case["samples"], first=64 + seed % 180)


def _run_ao(s):
    s["ao"].reset_sample()
    s["ao"].sample_count = s["first"]  # some way into the camera's samples
    for _ in range(s["samples"]):
        s["ao"].render()
    return s["ao"].image


def _prepare_path_trace(case, seed):
    P = _system([scenes.heightfield(case["size"], seed=seed)])
    vp, eye = _view(case, seed, (0.5, -0.35, 0.55), 45.0)
    lights = [pt.directional_light((3.0, 2.8, 2.5), (0.35, 0.25, -1.0)),
              pt.directional_light((1.0, 1.2, 1.5), (-0.4, 0.3, -0.8))][: case["lights"]]
    R = pt.DeviceReferencePathTracingRenderer(P, case["width"], case["height"], vp, eye, lights=lights,
                                              background_color=(0.4, 0.5, 0.7), max_path_depth=case["depth"],
                                              traversal=_traversal(case), schedule=case["schedule"], keep_radiance=True)
    return dict(kind="path_trace", P=P, R=R, samples=case["samples"])


def _run_path_trace(s):
    R = s["R"]
    R.reset_sample()
    for _ in range(s["samples"]):
        R.render()
    return dict(image=R.image, radiance=R.radiance)


# ---- rebuild -------------------------------------------------------------------------------------------------------

def _prepare_rebuild(case, seed):
    P = _system([_mesh(case, seed)])
    rays = _cuda_rays(_rays(case, seed))
    return dict(kind="rebuild", P=P, rays=rays, hits=torch.zeros((rays.shape[0], 4), device="cuda"))


def _run_rebuild(s):
    P = s["P"]
    P.build(blas_bin_size=4, device_build=True)
    P.trace(s["rays"], s["hits"])
    st = P.build_stats()
    return dict(_hit_outputs(s["hits"]), stats=[int(st[k]) for k in ("triangles", "nodes", "sah_splits", "median_fallbacks",
                                                                     "max_blas_depth", "device_bytes")])


# ---- queue primitives ----------------------------------------------------------------------------------------------

def _prepare_regroup(case, seed):
    n, L = case["count"], native.lib()
    g = torch.Generator(device="cuda").manual_seed(seed)
    bits = case["key_bits"]
    src = torch.randint(0, 1 << bits, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    size, most = C.c_size_t(), 0
    for f in (L.rdn_scan_scratch_size, L.rdn_compact_scratch_size, L.rdn_radix_sort_scratch_size):
        _ok(f(n, C.byref(size)))
        most = max(most, size.value)
    scratch = torch.empty(most + 256, dtype=torch.uint8, device="cuda")
    new = lambda k=n: torch.zeros(k, dtype=torch.int32, device="cuda")  # noqa: E731
    return dict(kind="regroup", n=n, bits=bits, src=src, iota=torch.arange(n, dtype=torch.int32, device="cuda"),
                flags=(torch.rand(n, generator=g, device="cuda") < 0.6).to(torch.int32), keys=new(), vals=new(),
                out=new(), count=new(1), sums=new(), scratch=scratch, ptr=(scratch.data_ptr() + 255) & ~255, bytes=most)


def _run_regroup(s):
    L, st, n = native.lib(), _stream(), s["n"]
    s["keys"].copy_(s["src"])
    s["vals"].copy_(s["iota"])
    _ok(L.rdn_radix_sort_u32(s["keys"].data_ptr(), s["vals"].data_ptr(), n, s["bits"], s["ptr"], s["bytes"], st))
    _ok(L.rdn_compact_u32(s["vals"].data_ptr(), s["flags"].data_ptr(), s["out"].data_ptr(), s["count"].data_ptr(), n,
                          s["ptr"], s["bytes"], st))
    _ok(L.rdn_scan_u32(s["flags"].data_ptr(), s["sums"].data_ptr(), n, 0, 0, s["ptr"], s["bytes"], st))
    return dict(keys=s["keys"], vals=s["vals"], kept=s["out"], count=s["count"], sums=s["sums"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _trace_work(rays, tris, io):
    """`rays` closest-hit queries: their records (io bytes a ray), the triangles and nodes they can touch (each once),
    and per ray two boxes a tree level and a leaf's four triangles."""
    touched = min(tris, 4 * rays)
    levels = math.log2(max(tris / 2, 2))
    return dict(bytes=rays * io + touched * (36 + 24), flops=rays * (levels * 2 * 24 + 4 * 45))


def _add(*works):
    return dict(bytes=sum(w["bytes"] for w in works), flops=sum(w["flops"] for w in works))


def work(case):
    kind = case["kind"]
    n = case.get("width", 0) * case.get("height", 0)
    if kind in ("query", "rebuild"):
        tris = case["size"] if case["mesh"] == "soup" else 2 * (case["size"] - 1) ** 2
        w = _trace_work(n, tris, 48 + (16 if case.get("context") else 0))
        if kind == "rebuild":
            # vertices and indices in; triangle records, both node layouts, the flat tree and the vertex copies out
            w = _add(w, dict(bytes=tris * (36 + 64 + 32 + 32 + 48 + 48 + 8), flops=tris * 21 * 30))
        return w
    if kind == "paths":
        tris, rays = (int(sum(x)) for x in _paths_sizes(case))
        return _trace_work(2 * rays, tris, 24 + 4)
    if kind == "path_loss":
        grids, counts = _path_loss_sizes(case)
        tris, rays = int(sum(2 * (grids - 1) ** 2)), int(sum(counts))
        seg = case["segments"]
        return _add(_trace_work(rays * seg, tris, 32 // seg + 8 + 4), dict(bytes=16 * int(sum(grids ** 2)),
                                                                         flops=rays * seg * 300))
    if kind == "regroup":
        return dict(bytes=36 * case["count"], flops=0)
    tris = 2 * (case["size"] - 1) ** 2
    if kind == "frame":
        return _trace_work(3 * n, tris, 11)
    if kind in ("loss", "hit_diff"):
        return _add(_trace_work(n, tris, 32 + 24 + 24 + 16), dict(bytes=16 * case["size"] ** 2, flops=n * 400))
    if kind == "ao":
        return _trace_work(2 * n * case["samples"], tris, 2)
    return _trace_work(n * case["samples"] * (1 + case["depth"]), tris, 8)


# ---- results in 64 bits --------------------------------------------------------------------------------------------

def _triangles64(mesh):
    p = torch.from_numpy(mesh.positions.astype(np.float64)).cuda()
    idx = torch.arange(p.shape[0], device="cuda") if mesh.indices is None else \
        torch.from_numpy(mesh.indices.astype(np.int64)).cuda()
    return p, idx.reshape(-1, 3)


def _first_hits64(p, idx, rays):
    """Index of the first triangle of each ray (-1: none), every triangle tried: the edge functions are linear in
    the ray's direction and moment, so that each is one matrix product."""
    o, d = rays[:, 0:3].double(), rays[:, 4:7].double()
    m = torch.cross(o, d, dim=1)
    v0, v1, v2 = (p[idx[:, k]] for k in range(3))
    e1, e2 = v1 - v0, v2 - v0
    nrm = torch.cross(e1, e2, dim=1)
    det_f = nrm.T.contiguous()
    # u (n . d) = -(d . (v0 x e2) + m . e2), v (n . d) = d . (v0 x e1) + m . e1, t (n . d) = n . v0 - n . o
    u_f = -torch.cat([torch.cross(v0, e2, dim=1), e2], 1).T.contiguous()
    v_f = torch.cat([torch.cross(v0, e1, dim=1), e1], 1).T.contiguous()
    c = (nrm * v0).sum(1)
    out = torch.empty(rays.shape[0], dtype=torch.int64, device="cuda")
    step = max(1, int(1e8) // idx.shape[0])
    for a in range(0, rays.shape[0], step):
        dd, mm, oo = d[a:a + step], m[a:a + step], o[a:a + step]
        inv = 1.0 / (dd @ det_f)
        dm = torch.cat([dd, mm], 1)
        u = (dm @ u_f).mul_(inv)
        v = (dm @ v_f).mul_(inv)
        bad = (u < 0) | (v < 0) | (u.add_(v) > 1)
        del u, v
        t = (c[None, :] - oo @ det_f).mul_(inv)
        bad |= ~(t >= 0)
        t.masked_fill_(bad, math.inf)
        best, at = t.min(1)
        out[a:a + step] = torch.where(torch.isfinite(best), at, -1)
    return out


def _solve64(p, idx, rays, tri):
    """t, u, v and what their gradients need, on the given triangles."""
    hit = tri >= 0
    k = idx[tri.clamp(min=0)]
    o, d = rays[:, 0:3].double(), rays[:, 4:7].double()
    v0, v1, v2 = (p[k[:, j]] for j in range(3))
    e1, e2, b = v1 - v0, v2 - v0, o - v0
    n = torch.cross(e1, e2, dim=1)
    det = -(d * n).sum(1)
    t = (b * n).sum(1) / det
    cu, cv = torch.cross(e2, -d, dim=1), torch.cross(-d, e1, dim=1)
    return hit, k, n, cu, cv, det, t, (b * cu).sum(1) / det, (b * cv).sum(1) / det


def _adjoint64(p, attr, sol, gt, gu, gv, ga):
    """Gradients of vertices (with the attribute), origins and directions for upstream gradients of t, u, v, value."""
    hit, k, n, cu, cv, det, t, u, v = sol
    a = attr.double()[k]
    gu, gv = gu + ga * (a[:, 1] - a[:, 0]), gv + ga * (a[:, 2] - a[:, 0])
    lam = (gt[:, None] * n + gu[:, None] * cu + gv[:, None] * cv) / det[:, None]
    lam[~hit] = 0
    grad = torch.zeros((p.shape[0], 4), dtype=torch.float64, device="cuda")
    for j, w in enumerate((1 - u - v, u, v)):
        g = torch.cat([-w[:, None] * lam, (w * ga)[:, None]], 1)
        g[~hit] = 0
        grad.index_add_(0, k[:, j], g)
    return grad, lam, t[:, None].masked_fill(~hit[:, None], 0) * lam


def exact(case, seed):
    if case["kind"] not in ("query", "loss", "hit_diff"):
        return None  # sampled images and paths, whole numbers
    if case["kind"] == "query":
        mesh = _mesh(case, seed)
        rays = _cuda_rays(_rays(case, seed))
    else:
        mesh, attr, rays, target = _field_and_target(case, seed)
    if rays.shape[0] * mesh.triangle_count > 4e10:
        return None  # every ray against every triangle takes too long
    p, idx = _triangles64(mesh)
    tri = _first_hits64(p, idx, rays)
    sol = _solve64(p, idx, rays, tri)
    hit, k, t, u, v = sol[0], sol[1], sol[6], sol[7], sol[8]
    if case["kind"] == "query":
        tuv = torch.stack([torch.where(hit, t, math.inf), torch.where(hit, u, 0.0), torch.where(hit, v, 0.0)], 1)
        return dict(tuv=tuv, prim=None, context=None)
    a = attr.double()[k]
    value = torch.where(hit, (1 - u - v) * a[:, 0] + u * a[:, 1] + v * a[:, 2], 0.0)
    if case["kind"] == "loss":
        off = torch.where(hit, value - target.double(), 0.0)
        zero = torch.zeros_like(off)
        grad, go, gd = _adjoint64(p, attr, sol, zero, zero, zero, 2 * off)
        return dict(loss=off.square().sum().reshape(1), value=value, tri=None, grad=grad, grad_origin=go,
                    grad_direction=gd)
    r = np.random.Generator(np.random.PCG64(seed + 29))
    g = torch.from_numpy(r.normal(size=(rays.shape[0], 4)).astype(np.float32)).cuda().double()
    grad, go, gd = _adjoint64(p, attr, sol, g[:, 0], g[:, 1], g[:, 2], g[:, 3])
    out = torch.stack([torch.where(hit, t, math.inf), torch.where(hit, u, 0.0), torch.where(hit, v, 0.0), value], 1)
    return dict(hit=out, tri=None, grad=grad, grad_origin=go, grad_direction=gd)
