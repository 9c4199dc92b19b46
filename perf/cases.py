"""The workloads this framework's speed is measured on, through its public entry points.

Kinds of work (the ranges are this repository's own: the configs of scenegen.py, the tests and
bench.py):

  rays      a batch of rays against a resident scene (RayQueue::traverse of the reference's tile
            scheduler, the server's ray batches): closest hits or occlusion, single-mesh and
            instanced scenes, with and without opacity masks, device buffers
  host_rays the same with rays and hits in host arrays (the reference's CPU traversal boundary)
  frame     one path-traced frame (PathTracer::render)
  vcm       one iteration of the VCM family (VCMIntegrator::render)
  grid      a photon hash grid built over a photon cloud and queried for the k nearest photons
            (HashGrid::build / query)
  build     a scene's BVHs built on the device (scene admission), then a first ray batch
  refit     a resident scene's BVHs refitted to moved vertices (animation), then a ray batch

Scenes are the repository's synthetic ones: `spheres` displaced spheres of 5,120 triangles each
over a ground quad with a two-triangle light (one mesh, one instance), or the instanced scene
(9 meshes, 201 instances, 1.3 M instanced triangles, five material kinds). A program keeps the
resident scene and the integrator; rays, seeds, views, photons and moved vertices are new inputs.
"""
import math

import numpy as np
import torch

from imbatracer_b200 import native as N
from imbatracer_b200 import scene as S
from imbatracer_b200 import scenegen as G
from imbatracer_b200.hashgrid import HashGrid
from imbatracer_b200.integrators import GpuScene, PathTracer, VcmIntegrator

T_FAR = 200.0   # rays end here: beyond every scene, and misses then report a finite distance


def listed():
    return [
        # One small tile of the reference's tile scheduler: launch latency counts.
        {"name": "rays_tile", "kind": "rays", "scene": "spheres", "spheres": 32, "rays": 2049, "any": False,
         "masked": False},
        # A serving ray batch over the instanced scene, incoherent directions, u and v wanted.
        {"name": "rays_instanced", "kind": "rays", "scene": "instanced", "spheres": 0, "rays": 1000003, "any": False,
         "masked": False},
        # Shadow rays towards the light through masked (foliage-like) geometry.
        {"name": "shadow_masked", "kind": "rays", "scene": "spheres", "spheres": 32, "rays": 2000000, "any": True,
         "masked": True},
        # The drop-in host boundary: the reference hands over host ray and hit arrays.
        {"name": "host_rays", "kind": "host_rays", "scene": "spheres", "spheres": 32, "rays": 250007, "any": False},
        # Config 1: an interactive preview frame.
        {"name": "frame_512", "kind": "frame", "scene": "spheres", "spheres": 32, "width": 512, "height": 512,
         "spp": 1, "path_len": 5, "rr_start": 0},
        # Config 2 at a quarter of its samples: a final-quality 1080p frame, 8 bounces.
        {"name": "frame_1080p", "kind": "frame", "scene": "instanced", "spheres": 0, "width": 1920, "height": 1080,
         "spp": 4, "path_len": 9, "rr_start": 3},
        # Config 3 at its own photon-grid parameters: 2 M triangles, 2^20 light paths, 720p.
        {"name": "vcm_720p", "kind": "vcm", "algo": "vcm", "spheres": 400, "width": 1280, "height": 720,
         "light_paths": 1 << 20, "path_len": 8, "knn": 10, "spec_grid": True},
        # A small bidirectional frame as the render server gets them.
        {"name": "bpt_small", "kind": "vcm", "algo": "bpt", "spheres": 8, "width": 200, "height": 152,
         "light_paths": 15200, "path_len": 8, "knn": 10, "spec_grid": False},
        # A small photon map with the reference's grid parameters (cell 2r, 2n buckets).
        {"name": "grid_small", "kind": "grid", "photons": 20011, "queries": 2000, "k": 16, "spec_grid": False},
        # The photon map of config 3: a query at every light vertex, k = 10, cell = r, 2^22 buckets.
        {"name": "grid_720p", "kind": "grid", "photons": 1740001, "queries": 1740001, "k": 10, "spec_grid": True},
        # Admission of the instanced scene to the server, up to its first ray batch.
        {"name": "build_instanced", "kind": "build", "scene": "instanced", "spheres": 0, "rays": 16384},
        # An animated 512k-triangle mesh: refit and one batch of rays per time step.
        {"name": "refit_spheres", "kind": "refit", "scene": "spheres", "spheres": 100, "rays": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "host_rays", "frame", "frame", "vcm", "vcm", "grid", "grid", "build", "refit"])
    scene = rng.choice(["spheres", "instanced"])
    spheres = _log(rng, 1, 100) if scene == "spheres" else 0
    if kind == "rays":
        masked = scene == "spheres" and rng.random() < 0.4
        return {"kind": kind, "scene": scene, "spheres": min(spheres, 40), "rays": _log(rng, 64, 2000000),
                "any": rng.random() < 0.5, "masked": masked}
    if kind == "host_rays":
        return {"kind": kind, "scene": scene, "spheres": min(spheres, 40), "rays": _log(rng, 64, 1000000),
                "any": rng.random() < 0.5}
    if kind == "frame":
        w, h, spp = _log(rng, 64, 1280), _log(rng, 64, 720), rng.choice([1, 2, 3, 4])
        return {"kind": kind, "scene": scene, "spheres": min(spheres, 40), "width": w, "height": h, "spp": spp,
                "path_len": rng.randint(2, 9), "rr_start": rng.choice([0, 3])}
    if kind == "vcm":
        return {"kind": kind, "algo": rng.choice(["vcm", "bpt", "ppm", "lt"]), "spheres": max(1, spheres),
                "width": 8 * _log(rng, 8, 120), "height": 8 * _log(rng, 8, 80), "light_paths": _log(rng, 2000, 700000),
                "path_len": rng.randint(3, 9), "knn": rng.choice([5, 10, 16]), "spec_grid": rng.random() < 0.3}
    if kind == "grid":
        return {"kind": kind, "photons": _log(rng, 1000, 1700000), "queries": _log(rng, 500, 1700000),
                "k": rng.choice([1, 8, 10, 16, 32, 48]), "spec_grid": rng.random() < 0.5}
    if kind == "build":
        return {"kind": kind, "scene": scene, "spheres": spheres, "rays": _log(rng, 1024, 65536)}
    return {"kind": "refit", "scene": scene, "spheres": spheres, "rays": _log(rng, 1024, 262144)}


# --------------------------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------------------------
_scenes = {}


def _desc(scene, spheres, masked=False):
    """A scene description, as a program has it after loading a file (kept between states)."""
    key = (scene, spheres, masked)
    if key not in _scenes:
        d = G.config2(1) if scene == "instanced" else G._sphere_field(1, max(1, spheres), 4, 512, 512, "field")
        if masked:
            rng = np.random.default_rng(5)
            mesh = d.meshes[0]
            mesh.texcoords = np.ascontiguousarray(mesh.vertices[:, [0, 2]] * np.float32(0.7) +
                                                  mesh.vertices[:, 1:2] * np.float32(0.3))
            n = len(d.materials)
            d.masks = np.zeros(n, N.MASK_DTYPE)
            d.masks["width"] = d.masks["height"] = 64
            d.masks["offset"] = 4 + 4096 * (np.arange(n) % 4)
            d.mask_buffer = np.concatenate([np.ones(4, np.uint8), (rng.random(4 * 4096) < 0.7).astype(np.uint8)])
            d.masks[n - 3:] = (1, 1, 0)     # the ground and the light stay opaque
        _scenes[key] = d
    return _scenes[key]


_host_trees = {}


def _tree(scene, spheres, masked=False):
    """The scene's host-built (spatial-split) trees: built or read once per program."""
    key = (scene, spheres, masked)
    if key not in _host_trees:
        d = _desc(*key)
        _host_trees[key] = S.build_traversal_data(d.meshes, d.instances, masks=d.masks, mask_buffer=d.mask_buffer)
    return _host_trees[key]


def _rays(desc, n, seed, to_light=False):
    """n rays with origins uniform in the scene's box (the field's, without the wide ground) and
    directions uniform on the sphere, or ending just before a point of the area light."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    rays[:, :3] = torch.rand((n, 3), generator=g, device="cuda") * 24 - 12
    if to_light:
        p = torch.rand((n, 3), generator=g, device="cuda")
        p = torch.stack([p[:, 0] * 6 - 3, torch.full_like(p[:, 0], 16.0), p[:, 2] * 6 - 3], 1)
        rays[:, 4:7] = p - rays[:, :3]
        rays[:, 3], rays[:, 7] = 1e-3, 1.0 - 1e-3
    else:
        d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
        rays[:, 4:7] = (d / d.norm(dim=1, keepdim=True)).float()
        rays[:, 3], rays[:, 7] = 0.0, T_FAR
    return rays


def _camera(desc, seed, w, h):
    r = np.random.default_rng(seed)
    c = desc.camera
    pos = tuple(float(x) for x in np.asarray(c.pos) + r.uniform(-0.5, 0.5, 3))
    return G.Camera(pos, c.dir, c.up, c.fov, w, h)


def _photons(n, seed):
    """Photons on surfaces, denser on top: 400 spheres of radius 0.5 to 2 and the ground below."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    centre, radius = u(400, 3) * 20 - 10, u(400) * 1.5 + 0.5
    pick = torch.multinomial(radius ** 2, n, replacement=True, generator=g)
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    d[:, 1] = torch.where(u(n) < 0.6, d[:, 1].abs(), d[:, 1])
    p = centre[pick] + d / d.norm(dim=1, keepdim=True) * radius[pick, None]
    ground = u(n) < 0.3
    spread = torch.randn((n, 2), generator=g, device="cuda", dtype=torch.float64) * 15
    on = torch.stack([spread[:, 0], torch.full_like(spread[:, 0], -10.0), spread[:, 1]], 1)
    return torch.where(ground[:, None], on, p).float().contiguous()


def _radius(case):
    """A merge radius that finds about ten photons on the average surface patch."""
    return float(math.sqrt(10.0 * 9000.0 / (math.pi * case["photons"])))


def _moved(desc, seed):
    """The scene's vertices at another time step: a smooth wave through every mesh."""
    r = np.random.default_rng(seed)
    k, ph = r.uniform(0.3, 0.9, 3), r.uniform(0, 6.28, 3)
    out = []
    for m in desc.meshes:
        v = m.vertices.astype(np.float64)
        out.append(np.ascontiguousarray(v + 0.1 * np.sin(v[:, [1, 2, 0]] * k + ph), np.float32))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("rays", "host_rays"):
        masked = case.get("masked", False)
        s["desc"] = desc = _desc(case["scene"], case["spheres"], masked)
        s["scene"] = S.DeviceScene(_tree(case["scene"], case["spheres"], masked))
        s["rays"] = _rays(desc, case["rays"], seed, to_light=case["any"])
        if kind == "host_rays":
            s["rays"] = s["rays"].cpu().numpy()
            s["hits"] = np.zeros((case["rays"], 4), np.int32)
        else:
            s["hits"] = torch.zeros((case["rays"], 4), dtype=torch.int32, device="cuda")
            s["v"] = None if case["any"] else torch.zeros(case["rays"], dtype=torch.float32, device="cuda")
    elif kind == "frame":
        desc = _desc(case["scene"], case["spheres"])
        s["scene"] = GpuScene(desc, td=_tree(case["scene"], case["spheres"]))
        s["pt"] = PathTracer(s["scene"], max_path_len=case["path_len"], rr_start=case["rr_start"])
        s["cam"] = _camera(desc, seed, case["width"], case["height"])
        s["seed"] = seed * 7919 + 1
    elif kind == "vcm":
        desc = _desc("spheres", case["spheres"])
        s["scene"] = GpuScene(desc, gpu_build=True)
        spec = case["spec_grid"]
        kw = {"base_radius": 0.8596, "radius_exponent": 1.0 / 3.0, "grid_cell_factor": 1.0,
              "grid_table_size": 1 << 22} if spec else {}
        s["vcm"] = VcmIntegrator(s["scene"], case["algo"], case["width"], case["height"], spp=1,
                                 max_path_len=case["path_len"], light_path_count=case["light_paths"],
                                 num_connections=1, num_knn=case["knn"],
                                 cam=_camera(desc, seed, case["width"], case["height"]), **kw)
        s["seed"] = seed * 7919 + 1
    elif kind == "grid":
        s["grid"] = HashGrid(0)
        s["photons"] = _photons(case["photons"], seed)
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        at = torch.randint(0, case["photons"], (case["queries"],), generator=g, device="cuda")
        off = torch.randn((case["queries"], 3), generator=g, device="cuda") * (0.1 * _radius(case))
        s["points"] = (s["photons"][at] + off).contiguous()
    elif kind == "build":
        desc = _desc(case["scene"], case["spheres"])
        s["meshes"] = [S.Mesh(v, m.indices, m.normals, m.texcoords, m.geom_normals)
                       for v, m in zip(_moved(desc, seed), desc.meshes)]
        s["instances"] = desc.instances
        s["rays"] = _rays(desc, case["rays"], seed)
        s["hits"] = torch.zeros((case["rays"], 4), dtype=torch.int32, device="cuda")
    elif kind == "refit":
        s["desc"] = desc = _desc(case["scene"], case["spheres"])
        s["scene"] = S.DeviceScene.build_gpu(desc.meshes, desc.instances)
        s["verts"] = torch.from_numpy(np.concatenate(_moved(desc, seed))).cuda()
        tv, off = [], 0
        for m in desc.meshes:
            t = np.zeros((m.triangle_count, 4), np.int32)
            t[:, :3] = m.indices[:, :3] + off
            tv.append(t)
            off += len(m.vertices)
        s["tri_verts"] = torch.from_numpy(np.concatenate(tv)).cuda()
        s["rays"] = _rays(desc, case["rays"], seed)
        s["hits"] = torch.zeros((case["rays"], 4), dtype=torch.int32, device="cuda")
    return s


# --------------------------------------------------------------------------------------------
# The work
# --------------------------------------------------------------------------------------------
def _hit_parts(hits):
    return {"tri": hits[:, 0], "inst": hits[:, 1], "t": hits[:, 2].view(torch.float32),
            "u": hits[:, 3].view(torch.float32)}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "rays":
        s["scene"].trace(s["rays"], s["hits"], any_hit=case["any"], v_out=s["v"])
        if case["any"]:
            return {"occluded": s["hits"][:, 0] >= 0}    # which occluder was met is not part of the answer
        return dict(_hit_parts(s["hits"]), v=s["v"])
    if kind == "host_rays":
        s["scene"].trace_host(s["rays"], s["hits"], any_hit=case["any"])
        if case["any"]:
            return {"occluded": s["hits"][:, 0] >= 0}
        h = s["hits"]
        return {"tri": h[:, 0], "inst": h[:, 1], "t": h[:, 2].view(np.float32), "u": h[:, 3].view(np.float32)}
    if kind == "frame":
        return s["pt"].render(case["spp"], s["seed"], case["width"], case["height"], cam=s["cam"], stats=False)
    if kind == "vcm":
        return s["vcm"].render(2, s["seed"], s["seed"] + 77, 0x9E3779B9)
    if kind == "grid":
        if case["spec_grid"]:
            s["grid"].build(s["photons"], _radius(case), 1.0, 1 << 22)
        else:
            s["grid"].build(s["photons"], _radius(case))
        ids, counts, d2 = s["grid"].query(s["points"], case["k"], with_d2=True)
        return {"ids": ids, "counts": counts, "d2": d2}
    if kind == "build":
        scene = S.DeviceScene.build_gpu(s["meshes"], s["instances"])
        scene.trace(s["rays"], s["hits"])
        return _hit_parts(s["hits"])
    lib = N.load()
    N.check(lib.imbart_scene_refit(s["scene"].handle, N.ptr(s["verts"]), s["verts"].shape[0], N.ptr(s["tri_verts"]),
                                   s["tri_verts"].shape[0], None), "imbart_scene_refit")
    s["scene"].trace(s["rays"], s["hits"])
    return _hit_parts(s["hits"])


# --------------------------------------------------------------------------------------------
# What the work cannot do without, and what its answers may differ by
# --------------------------------------------------------------------------------------------
def _scene_size(case):
    """(triangles, vertices, instances) of the case's scene."""
    if case.get("scene") == "instanced":
        d = _desc("instanced", 0)
        return (sum(m.triangle_count for m in d.meshes), sum(len(m.vertices) for m in d.meshes), len(d.instances))
    n = max(1, case["spheres"])
    return 5120 * n + 4, 2562 * n + 10, 1


def _ray_flops(tris, insts):
    # One 8-child node per level (six slab planes each, a multiply-add) and one triangle test.
    levels = math.log(max(tris, 8), 8) + (math.log(max(insts, 8), 8) if insts > 1 else 0)
    return levels * 8 * 6 * 2 + 60


def work(case):
    kind = case["kind"]
    if kind == "grid":
        n, q, k = case["photons"], case["queries"], case["k"]
        return {"bytes": 12 * n + 12 * q + q * (8 * k + 4), "flops": 8.0 * q * k}
    tris, verts, insts = _scene_size(case)
    scene = 12 * verts + 12 * tris + 64 * insts
    per = _ray_flops(tris, insts)
    if kind in ("rays", "host_rays"):
        n = case["rays"]
        out = 1 if case["any"] else 16
        return {"bytes": n * (32 + out) + scene, "flops": n * per}
    if kind in ("build", "refit"):
        n = case["rays"]
        return {"bytes": scene + 48 * tris + 48 * n, "flops": n * per + tris * 30.0}
    px = case["width"] * case["height"]
    if kind == "frame":
        # Every sample is at least one closest-hit and one shadow ray.
        n = px * case["spp"]
        return {"bytes": scene + 12 * px, "flops": 2.0 * n * per}
    n = (0 if case["algo"] == "lt" else px) + case["light_paths"]
    cache = 0 if case["algo"] == "lt" else 2 * 112 * case["light_paths"]
    return {"bytes": scene + 12 * px + cache, "flops": 2.0 * n * per}


def tolerance(case):
    kind = case["kind"]
    if kind in ("frame", "vcm"):
        # The order of 32-bit additions into a pixel.
        return {"rel": 1e-5}
    if kind == "grid":
        # Photons at equal squared distances at the end of a full list: either may be kept.
        return {"rel": 1e-6, "differ": 1e-4}
    return "exact"   # hits do not depend on the tree or the order of the tests


def _closest64(rays, corners, ids=None):
    """Closest hits by brute force in 64 bits: (t, u, v) per ray (t_max, 0, 0 for a miss).
    corners: (n, 3, 3) world-space triangles."""
    r = rays.double()
    org, dirn, tmin, tmax = r[:, :3], r[:, 4:7], r[:, 3], r[:, 7]
    best = tmax.clone()
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    a, e1, e2 = corners[:, 0], corners[:, 1] - corners[:, 0], corners[:, 2] - corners[:, 0]
    step = max(1, (1 << 24) // max(1, len(r)))
    for at in range(0, len(a), step):
        x, y, z = a[at:at + step], e1[at:at + step], e2[at:at + step]
        p = torch.linalg.cross(dirn[:, None, :], z[None, :, :])
        det = (p * y[None]).sum(-1)
        tv = org[:, None, :] - x[None]
        u = (tv * p).sum(-1) / det
        q = torch.linalg.cross(tv, y[None].expand_as(tv))
        v = (q * dirn[:, None, :]).sum(-1) / det
        t = (q * z[None]).sum(-1) / det
        bad = ~((u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin[:, None]))
        t = t.masked_fill(bad, math.inf)
        m, i = t.min(1)
        take = m < best
        best = torch.where(take, m, best)
        bu = torch.where(take, u.gather(1, i[:, None])[:, 0], bu)
        bv = torch.where(take, v.gather(1, i[:, None])[:, 0], bv)
    return best, bu, bv


def _corners(meshes, instances):
    out = []
    for inst in instances:
        m = meshes[inst.mesh_id]
        v = torch.from_numpy(m.vertices).cuda().double()
        mat = torch.from_numpy(np.ascontiguousarray(inst.mat[:3])).cuda().double()
        v = v @ mat[:, :3].T + mat[:, 3]
        out.append(v[torch.from_numpy(np.ascontiguousarray(m.indices[:, :3])).cuda().long()])
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        if case["photons"] * case["queries"] > 2e9:
            return None
        p = _photons(case["photons"], seed)
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        at = torch.randint(0, case["photons"], (case["queries"],), generator=g, device="cuda")
        off = torch.randn((case["queries"], 3), generator=g, device="cuda") * (0.1 * _radius(case))
        q = (p[at] + off).double()
        pd, r2, k = p.double(), _radius(case) ** 2, case["k"]
        rows = []
        for c in q.split(max(1, (1 << 24) // len(pd))):
            d = ((c[:, None, :] - pd[None]) ** 2).sum(-1).topk(min(k, len(pd)), largest=False).values
            rows.append(torch.where(d <= r2, d, torch.zeros_like(d)))
        return {"ids": None, "counts": None, "d2": torch.cat(rows)}
    if kind in ("rays", "host_rays", "build", "refit"):
        if case.get("any") or case.get("masked"):
            return None
        tris = 1300000 if case["scene"] == "instanced" else 5120 * max(1, case["spheres"])
        if tris * case["rays"] > 4e10:
            return None
        desc = _desc(case["scene"], case["spheres"])
        meshes = desc.meshes
        if kind in ("build", "refit"):
            meshes = [S.Mesh(v, m.indices, m.normals, m.texcoords, m.geom_normals)
                      for v, m in zip(_moved(desc, seed), desc.meshes)]
        t, u, v = _closest64(_rays(desc, case["rays"], seed), _corners(meshes, desc.instances))
        out = {"tri": None, "inst": None, "t": t, "u": u}
        return dict(out, v=v) if kind == "rays" else out
    return None   # a whole light-transport run has no 64-bit value at hand
