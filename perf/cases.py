"""Timed cases of the ray tracer: what a program has it do, through its public calls.

A case is a plain dict; `kind` names the call sequence and the other keys its
sizes and options.  The kinds:

  frame      one frame of an animation or of a static scene: (deform the mesh,)
             rebuild the grid, trace every pixel's ray and its shadow ray
  frame_host the same frame for a host program: keyframe staged from pinned
             host memory, rebuild, hits and occlusion back in pinned memory
  diffuse    rebuild, camera rays with one diffuse secondary ray each, and the
             closest hits of those secondary rays (the skewed-density scene)
  build      the grid build alone, to completion: offsets, lists, records
  rays       closest hits or occlusion of a ray array in device memory
  rays_host  the same for arrays in host memory, copies included
  batch      many uneven scenes built and traced together
  instances  camera rays over placed instances of a few scenes
  render     a shaded frame: shadows, reflection, refraction

Geometry is seeded and synthetic, in the shapes the framework's own workloads
use: a deforming UV sphere, a ground plane under debris, a scene of skewed
density, and small triangle soups.
"""
import collections
import math
import os
import sys
import zlib

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("grid-rt_gb300"))

from gridrt import lib, scenes  # noqa: E402

Camera = collections.namedtuple("Camera", "eye base_dir near_u near_v width height")

EPS = 2e-4                      # the rays' tnear
FLT_MAX = float(np.finfo(np.float32).max)
PLANE_LIGHT = (2.0, 4.0, 2.0)
SPHERE_LIGHT = (3.0, 4.0, 2.0)
VIEW = {"plane": ((0.0, 1.5, 3.0), (0.0, 0.3, 0.0)),
        "sphere": ((1.6, 1.2, 2.4), (0.0, 0.0, 0.0)),
        "skewed": ((0.9, 0.6, 1.5), (0.0, 0.0, 0.0))}
BACKGROUND = (0.9, 0.95, 1.0)
LIGHTS = (((2.0, 4.0, 2.0), (0.8, 0.8, 0.8), True), ((-3.0, 2.0, 1.0), (0.3, 0.3, 0.4), False))
# type, ambient, diffuse, specular exponent, reflexion, refraction index, opacity
MATERIALS = ((lib.RTG_MAT_PHONG, 0.2, (1.0, 1.0, 1.0), 32.0, 0.35, 1.0, 1.0),
             (lib.RTG_MAT_PHONG_COLOR, 0.2, (0.8, 0.3, 0.2), 32.0, 0.0, 1.3, 0.6),
             (lib.RTG_MAT_HEADLIGHT, 0.1, (1.0, 1.0, 1.0), 32.0, 0.0, 1.0, 1.0),
             (lib.RTG_MAT_HEADLIGHT_COLOR, 0.1, (0.2, 0.6, 0.9), 32.0, 0.0, 1.0, 1.0))


def listed():
    return [
        # a handful of triangles rebuilt alone, as for a gizmo or a test scene: latency and launches
        dict(name="build_tiny", kind="build", mesh="soup", tris=500, k=6, records=False),
        # a large static scene's load-time build at the reference's density
        dict(name="build_large", kind="build", mesh="plane", tris=1000000, k=6, records=False),
        # a picking or visibility query from host code: few rays, host arrays
        dict(name="rays_host_small", kind="rays_host", tris=10001, rays=4097, mode="nearest", k=4),
        # the deforming mesh of the headline benchmark, a 1024 x 1024 frame
        dict(name="frame_sphere", kind="frame", mesh="sphere", lat=160, lon=320, width=1024, height=1024,
             order="morton8", k=4, records=False),
        # the same frames driven by a host program
        dict(name="frame_host_sphere", kind="frame_host", lat=160, lon=320, width=1024, height=1024,
             order="morton8", k=4),
        # the plain method's scene: plane and debris, 512 x 512
        dict(name="frame_plane", kind="frame", mesh="plane", tris=65536, width=512, height=512,
             order="scanline", k=4, records=False),
        # a million triangles, nine tenths of them in one small box; incoherent secondary rays
        dict(name="diffuse_skewed", kind="diffuse", tris=1048576, width=1024, height=1024, order="morton8",
             k=2, records=True),
        # a serving request's closest-hit rays: incoherent, many
        dict(name="rays_nearest_large", kind="rays", tris=495000, rays=4000000, mode="nearest", k=4, records=False),
        # visibility segments between random points, an odd count
        dict(name="rays_any", kind="rays", tris=120011, rays=700001, mode="any", k=4, records=False),
        # many uneven scenes, each with its own rays
        dict(name="batch_64", kind="batch", scenes=64, tris=100000, rays=300000, k=2),
        # two-level scene: sixteen placed instances of three meshes
        dict(name="instances_16", kind="instances", instances=16, tris=65536, width=1024, height=1024),
        # a shaded frame with two lights, reflection and refraction
        dict(name="render_640", kind="render", tris=24577, width=640, height=480, depth=3, k=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "rays", "rays_host", "frame", "frame", "frame_host", "diffuse", "batch",
                       "instances", "render"])
    k = rng.choice([2, 3, 4, 6, 8])
    if kind == "build":
        mesh = rng.choice(["soup", "plane", "skewed"])
        return dict(kind=kind, mesh=mesh, tris=_log(rng, 100, 3000) if mesh == "soup" else _log(rng, 2000, 1000000),
                    k=k, records=rng.random() < 0.3)
    if kind == "rays":
        return dict(kind=kind, tris=_log(rng, 5000, 495000), rays=_log(rng, 30000, 4000000),
                    mode=rng.choice(["nearest", "any"]), k=k, records=rng.random() < 0.3)
    if kind == "rays_host":
        return dict(kind=kind, tris=_log(rng, 1000, 60000), rays=_log(rng, 500, 300000),
                    mode=rng.choice(["nearest", "any"]), k=k)
    if kind in ("frame", "frame_host"):
        mesh = rng.choice(["sphere", "plane"]) if kind == "frame" else "sphere"
        order = rng.choice(["scanline", "morton8"])
        step = 8 if order == "morton8" else 1
        size = dict(width=_log(rng, 160, 1024) // step * step, height=_log(rng, 160, 1024) // step * step,
                    order=order, k=k)
        if mesh == "sphere":
            lat = _log(rng, 24, 160)
            d = dict(kind=kind, mesh=mesh, lat=lat, lon=2 * lat + rng.randrange(-3, 4), **size)
        else:
            d = dict(kind=kind, mesh=mesh, tris=_log(rng, 2000, 300000), **size)
        if kind == "frame_host":
            del d["mesh"]
        else:
            d["records"] = rng.random() < 0.3
        return d
    if kind == "diffuse":
        return dict(kind=kind, tris=_log(rng, 60000, 1048576), width=8 * _log(rng, 30, 128),
                    height=8 * _log(rng, 30, 128), order=rng.choice(["scanline", "morton8"]), k=rng.choice([2, 4]),
                    records=rng.random() < 0.7)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randrange(3, 65), tris=_log(rng, 5000, 100000),
                    rays=_log(rng, 10000, 300000), k=rng.choice([2, 4]))
    if kind == "instances":
        return dict(kind=kind, instances=rng.randrange(2, 33), tris=_log(rng, 2000, 65536),
                    width=_log(rng, 200, 1024), height=_log(rng, 200, 1024))
    return dict(kind=kind, tris=_log(rng, 4000, 60000), width=_log(rng, 160, 640), height=_log(rng, 120, 480),
                depth=rng.randrange(0, 4), k=k)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(case, seed):
    text = ",".join("%s=%s" % (k, case[k]) for k in sorted(case) if k != "name")
    return np.random.default_rng([int(seed), zlib.crc32(text.encode())])


def _plane(rng, tris):
    """A ground plane of about half the triangles under debris."""
    quads = max(2, int(round(math.sqrt(tris / 4.0))))
    return scenes.plane_and_debris(int(rng.integers(1 << 31)), quads, max(1, tris - 2 * quads * quads))


def _soup(rng, tris):
    return scenes.tiny_scene(int(rng.integers(1 << 31)), tris)


def _mesh(case, rng):
    mesh = case["mesh"]
    if mesh == "plane":
        s = _plane(rng, case["tris"])
    elif mesh == "skewed":
        s = scenes.skewed_density(int(rng.integers(1 << 31)), case["tris"])
    else:
        s = _soup(rng, case["tris"])
    return s.verts, s.idx


def _build_mesh(case, seed):
    """The same triangles for every seed, so that every grid has the same size;
    the seed says which of them comes first and which corner of each."""
    verts, idx = _mesh(case, _rng(case, 0))
    rng = _rng(case, seed)
    turn = (np.arange(3) + rng.integers(0, 3, size=(idx.shape[0], 1))) % 3
    return verts, np.ascontiguousarray(np.roll(np.take_along_axis(idx, turn, 1), int(rng.integers(idx.shape[0])), 0))


def _camera(view, width, height):
    c = scenes.look_at_camera(VIEW[view][0], VIEW[view][1], (0.0, 1.0, 0.0), 60.0, width, height)
    return Camera(c.eye, c.base_dir, c.near_u, c.near_v, width, height)


def _random_rays(rng, n, lo, hi, segments):
    """Origins anywhere in the box, directions anywhere; or segments between two points of the box."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    lo, hi = (torch.tensor(np.asarray(x, np.float32), device="cuda") for x in (lo, hi))
    r = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    if segments:
        r[:, 4:7] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda") - r[:, 0:3]
    else:
        d = torch.randn((n, 3), generator=g, device="cuda")
        r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    d = r[:, 4:7]
    d[d == 0] = 1e-7
    r[:, 3] = EPS
    r[:, 7] = 1.0 if segments else FLT_MAX
    return r


def _hits(n, pinned=False):
    """An output buffer of n hits, and the same memory as ids and as (t, u, v)."""
    h = torch.zeros((n, 4), dtype=torch.int32, device="cpu" if pinned else "cuda", pin_memory=pinned)
    return h, {"id": h[:, 0], "tuv": h.view(torch.float32)[:, 1:]}


class _Device:
    """Device memory of a scene as a tensor, which keeps the scene alive."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}


def _as_tensor(owner, ptr, shape, kind):
    return torch.as_tensor(_Device(owner, ptr, shape, kind), device="cuda")


def _scene(verts, idx, k, records=False):
    s = lib.Scene(0)
    if records:
        s.set_tuning(cell_records=True)
    s.set_geometry(verts, idx)
    s.build(k)
    return s


def _transform(rng):
    """World-from-local and its inverse: a rotation, a uniform scale, a translation."""
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                  [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                  [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
    s, t = rng.uniform(0.4, 1.2), rng.uniform(-3.0, 3.0, size=3)
    inv = np.concatenate([R.T / s, (-(R.T / s) @ t)[:, None]], axis=1)
    return np.concatenate([s * R, t[:, None]], axis=1).astype(np.float32), inv.astype(np.float32)


def _instance_inputs(case, rng):
    lat = max(8, int(round(math.sqrt(case["tris"] / 4.0))))
    v, i, _ = scenes.sphere_mesh(lat, 2 * lat)
    p = _plane(rng, case["tris"])
    s = _soup(rng, max(100, case["tris"] // 4))
    meshes = [(v, i), (p.verts, p.idx), (s.verts, s.idx)]
    placed = [(j % 3, *_transform(rng)) for j in range(case["instances"])]
    c = scenes.look_at_camera((5.0, 4.0, 7.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 60.0, case["width"], case["height"])
    return meshes, placed, Camera(c.eye, c.base_dir, c.near_u, c.near_v, case["width"], case["height"])


def _camera_rays(cam):
    """Scanline pixel-centre rays of a camera, on the device."""
    i = torch.arange(cam.width * cam.height, device="cuda")
    us = ((i % cam.width).float() + 0.5) / cam.width
    vs = (torch.div(i, cam.width, rounding_mode="floor").float() + 0.5) / cam.height
    r = torch.empty((i.numel(), 8), dtype=torch.float32, device="cuda")
    for a in range(3):
        r[:, a] = float(cam.eye[a])
        r[:, 4 + a] = float(cam.base_dir[a]) + float(cam.near_u[a]) * us + float(cam.near_v[a]) * vs
    r[:, 3], r[:, 7] = EPS, FLT_MAX
    return r


def _batch_inputs(case, rng):
    """Scenes of log-uniform sizes, the same for every seed; per scene 60% camera
    rays and 40% random ones for closest hits, and for every fourth scene
    occlusion segments too."""
    items, sizes = [], _rng(case, 0)
    for j in range(case["scenes"]):
        sc = _plane(rng, int(round(math.exp(sizes.uniform(math.log(1000), math.log(case["tris"]))))))
        n = int(round(math.exp(sizes.uniform(math.log(4000), math.log(case["rays"])))))
        side = max(8, int(math.sqrt(0.6 * n)))
        lo, hi = sc.verts.min(axis=0), sc.verts.max(axis=0)
        rays = torch.cat([_camera_rays(_camera("plane", side, side)),
                          _random_rays(rng, max(1, n - side * side), lo, hi, False)])
        seg = _random_rays(rng, max(1, n // 4), lo, hi, True) if j % 4 == 3 else None
        items.append((sc, rays, seg))
    return items


def _render_inputs(case, rng):
    sc = _plane(rng, case["tris"])
    v, f = sc.verts.astype(np.float64), sc.idx
    fn = np.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])
    nrm = np.zeros_like(v)
    for a in range(3):
        np.add.at(nrm, f[:, a], fn)
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-30)
    colors = rng.uniform(0.2, 1.0, size=v.shape)
    mat = rng.integers(0, 4, size=f.shape[0]).astype(np.int32)
    mat[v[f[:, 0], 1] == 0] = 0                       # the ground reflects
    return sc, nrm.astype(np.float32), colors.astype(np.float32), mat, _camera("plane", case["width"], case["height"])


def prepare(case, seed):
    rng, kind, st = _rng(case, seed), case["kind"], {"case": case}
    if kind in ("frame", "frame_host"):
        sphere = kind == "frame_host" or case["mesh"] == "sphere"
        st["cam"] = _camera("sphere" if sphere else "plane", case["width"], case["height"])
        st["light"] = np.array(SPHERE_LIGHT if sphere else PLANE_LIGHT, np.float32)
        n = case["width"] * case["height"]
        host = kind == "frame_host"
        st["hits"], st["out"] = _hits(n, pinned=host)
        st["out"]["occluded"] = st["occ"] = torch.zeros(n, dtype=torch.uint8, device="cpu" if host else "cuda",
                                                        pin_memory=host)
        if sphere:
            verts, idx, nrm = scenes.sphere_mesh(case["lat"], case["lon"])
            st["phase"] = float(np.float32(rng.uniform(0.0, 6.0)))
            if host:
                moved = _deformed(verts, nrm, st["phase"]).astype(np.float32)
                st["key"] = torch.from_numpy(moved).pin_memory()
                st["copy"] = torch.cuda.Stream()
                verts = moved
            else:
                st["base"], st["nrm"] = torch.from_numpy(verts).cuda(), torch.from_numpy(nrm).cuda()
        else:
            verts, idx = _mesh(case, rng)
        st["scene"] = _scene(verts, idx, case["k"], case.get("records", False))
        # room for the deformed frames' grids, as an animation reserves it
        info = st["scene"].info()
        st["scene"].reserve(info["ncells"] * 5 // 4, info["nrefs"] * 5 // 4)
        st["scene"].build(case["k"])
    elif kind == "diffuse":
        st["seed"] = int(rng.integers(1 << 62))
        s = scenes.skewed_density(int(rng.integers(1 << 31)), case["tris"])
        st["cam"] = _camera("skewed", case["width"], case["height"])
        n = st["n"] = case["width"] * case["height"]
        st["hits"], o1 = _hits(n)
        st["hits2"], o2 = _hits(n)
        st["rays"] = torch.empty((n, 8), dtype=torch.float32, device="cuda")
        st["out"] = {"primary": o1, "secondary": o2, "rays": st["rays"]}
        st["scene"] = _scene(s.verts, s.idx, case["k"], case["records"])
    elif kind == "build":
        verts, idx = _build_mesh(case, seed)
        s = st["scene"] = _scene(verts, idx, case["k"], case["records"])
        s.build(case["k"])
        info = s.info()
        off, ids, tri = s.device_arrays()
        st["out"] = {"offsets": _as_tensor(s, off, (info["ncells"] + 1,), "<i4"),
                     "ids": _as_tensor(s, ids, (info["nrefs"],), "<i4"),
                     "records": _as_tensor(s, tri, (idx.shape[0], 3, 4), "<f4")[:, :, :3]}
    elif kind in ("rays", "rays_host"):
        s = _plane(rng, case["tris"])
        st["scene"] = _scene(s.verts, s.idx, case["k"], case.get("records", False))
        n, seg = case["rays"], case["mode"] == "any"
        st["rays"] = _random_rays(rng, n, s.verts.min(axis=0), s.verts.max(axis=0), seg)
        if kind == "rays_host":
            st["rays"] = st["rays"].cpu().numpy()
        elif seg:
            st["occ"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        else:
            st["hits"], st["out"] = _hits(n)
    elif kind == "batch":
        items = _batch_inputs(case, rng)
        st["scenes"], tasks = [], []
        n, m = sum(len(r) for _, r, _ in items), sum(len(g) for _, _, g in items if g is not None)
        st["hits"], st["out"] = _hits(n)
        st["out"]["occluded"] = st["occ"] = torch.zeros(m, dtype=torch.uint8, device="cuda")
        i = j = 0
        for t, (sc, rays, seg) in enumerate(items):
            s = lib.Scene(0)
            s.set_geometry(sc.verts, sc.idx)
            st["scenes"].append(s)
            tasks.append((t, lib.RTG_MODE_NEAREST, rays, len(rays), st["hits"][i:]))
            i += len(rays)
            if seg is not None:
                tasks.append((t, lib.RTG_MODE_ANY, seg, len(seg), st["occ"][j:]))
                j += len(seg)
        st["batch"] = lib.Batch(st["scenes"], [case["k"]] * len(items), tasks)
    elif kind == "instances":
        meshes, placed, cam = _instance_inputs(case, rng)
        st["scenes"] = [_scene(v, i, 4) for v, i in meshes]
        st["set"] = lib.Instances([(st["scenes"][m], a, b) for m, a, b in placed])
        st["rays"], st["n"] = _camera_rays(cam), cam.width * cam.height
        st["hits"], st["out"] = _hits(st["n"])
        st["out"]["instance"] = st["inst"] = torch.zeros(st["n"], dtype=torch.int32, device="cuda")
    else:
        sc, nrm, colors, mat, st["cam"] = _render_inputs(case, rng)
        st["scene"] = _scene(sc.verts, sc.idx, case["k"])
        st["nrm"], st["colors"], st["mat"] = (torch.from_numpy(x).cuda() for x in (nrm, colors, mat))
        st["mats"] = [lib.material(t, ambient=(a,) * 3, diffuse=d, specular_exponent=e, reflexion=r,
                                   refraction_index=i, opacity=o) for t, a, d, e, r, i, o in MATERIALS]
        st["lights"] = [lib.point_light(*x) for x in LIGHTS]
        st["rgb"] = torch.zeros((case["width"] * case["height"], 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "frame":
        s = st["scene"]
        if "base" in st:
            s.deform(st["base"], st["nrm"], 0.05, 3.0, st["phase"])
        s.build_async(case["k"])
        s.trace_frame_device(st["cam"], st["light"], st["hits"], st["occ"], None, order=case["order"])
        return st["out"]
    if kind == "frame_host":
        s = st["scene"]
        s.stage_vertices(st["key"], st["key"].shape[0], st["copy"].cuda_stream)
        s.build_async(case["k"])
        s.trace_frame_wait(s.trace_frame_async(st["cam"], st["light"], st["hits"], st["occ"], order=case["order"]))
        return st["out"]
    if kind == "diffuse":
        s = st["scene"]
        s.build_async(case["k"])
        s.trace_camera_diffuse_device(st["cam"], st["seed"], st["hits"], st["rays"], order=case["order"])
        s.trace_nearest_device(st["rays"], st["n"], st["hits2"])
        return st["out"]
    if kind == "build":
        st["scene"].build(case["k"])
        return st["out"]
    if kind == "rays":
        if case["mode"] == "any":
            st["scene"].trace_any_device(st["rays"], case["rays"], st["occ"])
            return st["occ"]
        st["scene"].trace_nearest_device(st["rays"], case["rays"], st["hits"])
        return st["out"]
    if kind == "rays_host":
        if case["mode"] == "any":
            return st["scene"].trace_any(st["rays"])
        h = st["scene"].trace_nearest(st["rays"])
        return {"id": h.view(np.int32)[:, 0], "tuv": h[:, 1:]}
    if kind == "batch":
        st["batch"].build_async()
        st["batch"].trace_async()
        return st["out"]
    if kind == "instances":
        st["set"].trace_nearest_device(st["rays"], st["n"], st["hits"], st["inst"])
        return st["out"]
    rays = st["scene"].render(st["cam"], st["nrm"], st["mats"], st["lights"], st["rgb"], d_colors=st["colors"],
                              d_material=st["mat"], background=BACKGROUND, max_depth=case["depth"])
    return {"rgb": st["rgb"], "rays": rays}


def work(case):
    """Bytes of the vertices, indices, rays and results, each once; for flops one
    triangle test (45) a ray, and for a build one box (40) a triangle."""
    kind, k = case["kind"], case.get("k", 4)
    if kind in ("frame", "frame_host") and "lat" in case:
        tris, verts = 2 * case["lat"] * case["lon"], (case["lat"] + 1) * case["lon"]
    elif kind == "batch":
        tris = case["scenes"] * (case["tris"] - 1000) / math.log(case["tris"] / 1000)
        verts = 1.75 * tris
    else:
        tris = case["tris"]
        verts = 3 * tris if kind == "diffuse" or case.get("mesh") in ("soup", "skewed") else 1.75 * tris
    geo, grid = 12 * verts + 12 * tris, 4 * k * tris + 8 * tris    # offsets and about two references a triangle
    n = case.get("width", 0) * case.get("height", 0)
    if kind == "build":
        return {"bytes": geo + grid + 48 * tris, "flops": 40 * tris}
    if kind == "frame":
        return {"bytes": geo * (2 if "lat" in case else 1) + grid + 17 * n, "flops": 90 * n + 40 * tris}
    if kind == "frame_host":
        return {"bytes": geo + grid + 17 * n, "flops": 90 * n + 40 * tris}
    if kind == "diffuse":
        return {"bytes": geo + grid + 64 * n, "flops": 90 * n + 40 * tris}
    if kind in ("rays", "rays_host"):
        n = case["rays"]
        return {"bytes": grid + 36 * tris + n * (33 if case["mode"] == "any" else 48), "flops": 45 * n}
    if kind == "batch":
        n = case["scenes"] * (case["rays"] - 4000) / math.log(case["rays"] / 4000)
        return {"bytes": geo + grid + 48 * n + 33 * n / 16, "flops": 48 * n + 40 * tris}
    if kind == "instances":
        return {"bytes": 2.25 * (grid + 36 * tris) + 52 * n, "flops": 45 * n}
    return {"bytes": grid + 36 * tris + 12 * n, "flops": 120 * n}


# ---------------------------------------------------------------------------
# the same in 64 bits, by testing every triangle
# ---------------------------------------------------------------------------
TESTS = 2.5e10                # ray-triangle tests that fit the time


def _deformed(verts, nrm, phase):
    v = verts.astype(np.float64)
    return v + (0.05 * np.sin(3.0 * v[:, :1] + phase)) * nrm.astype(np.float64)


def _t64(x):
    return torch.as_tensor(np.asarray(x, np.float64), device="cuda")


def _tri64(verts, idx):
    v = verts if isinstance(verts, torch.Tensor) else _t64(verts)
    f = torch.as_tensor(np.asarray(idx, np.int64), device="cuda")
    return v[f[:, 0]], v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]]


def _closest(o, d, tri, lo=EPS / 2, hi=math.inf):
    """(triangle or -1, t, u, v) of the nearest hit of every ray, by Moller-Trumbore
    written as products of ray and triangle vectors."""
    v0, e1, e2 = tri
    n = torch.linalg.cross(e1, e2)
    ray = torch.cat([torch.linalg.cross(o, d), d, o, torch.ones_like(o[:, :1])], 1)
    z = torch.zeros_like(e1)
    U = torch.cat([e2, -torch.linalg.cross(e2, v0)], 1).T.contiguous()
    V = torch.cat([-e1, -torch.linalg.cross(v0, e1)], 1).T.contiguous()
    T = torch.cat([n, -(v0 * n).sum(1, keepdim=True)], 1).T.contiguous()
    D = -n.T.contiguous()
    R, N = len(o), len(v0)
    out = (torch.full((R,), -1, dtype=torch.int64, device="cuda"),) + tuple(
        torch.zeros(R, dtype=torch.float64, device="cuda") for _ in range(3))
    if N == 0:
        return out
    step = max(1, int(8e7 // N))
    for a in range(0, R, step):
        r = ray[a:a + step]
        inv = 1.0 / (r[:, 3:6] @ D)
        u, v, t = (r[:, :6] @ U) * inv, (r[:, :6] @ V) * inv, (r[:, 6:] @ T) * inv
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t >= lo) & (t < hi), t, math.inf)
        m, j = t.min(1)
        hit = torch.isfinite(m)
        at = j[:, None]
        out[0][a:a + step] = torch.where(hit, j, -1)
        for x, y in zip(out[1:], (m, u.gather(1, at)[:, 0], v.gather(1, at)[:, 0])):
            x[a:a + step] = torch.where(hit, y, 0.0)
    return out


def _pixel_order(cam, order):
    """Scanline index of ray i."""
    i = torch.arange(cam.width * cam.height, device="cuda")
    if order == "scanline":
        return i
    tile, r = i // 64, i % 64
    x = tile % (cam.width // 8) * 8 + (r & 1 | r >> 1 & 2 | r >> 2 & 4)
    y = tile // (cam.width // 8) * 8 + (r >> 1 & 1 | r >> 2 & 2 | r >> 3 & 4)
    return y * cam.width + x


def _camera64(cam):
    i = torch.arange(cam.width * cam.height, device="cuda", dtype=torch.float64)
    us, vs = (torch.remainder(i, cam.width) + 0.5) / cam.width, (torch.floor(i / cam.width) + 0.5) / cam.height
    d = _t64(cam.base_dir) + us[:, None] * _t64(cam.near_u) + vs[:, None] * _t64(cam.near_v)
    return _t64(cam.eye).expand(len(d), 3).contiguous(), d


def _camera_hits(cam, tri):
    """_closest for a camera's rays, in scanline order: the image in tiles, each
    against the triangles whose projection meets it."""
    o, d = _camera64(cam)
    eye = _t64(cam.eye)
    v0, e1, e2 = (x.clone() for x in tri)
    v0 -= eye
    M = torch.linalg.inv(torch.stack([_t64(cam.near_u), _t64(cam.near_v), _t64(cam.base_dir)], 1))
    c = torch.stack([v0, v0 + e1, v0 + e2], 1) @ M.T             # (u t, v t, t) of the corners
    front = (c[:, :, 2] > 1e-3).all(1)
    p = c[:, :, :2] / torch.where(front[:, None, None], c[:, :, 2:], torch.ones_like(c[:, :, 2:]))
    lo, hi = p.min(1).values, p.max(1).values
    lo[~front], hi[~front] = -math.inf, math.inf
    lo[(c[:, :, 2] < 0).all(1)] = math.inf                        # behind the eye
    n = cam.width * cam.height
    out = [torch.full((n,), -1, dtype=torch.int64, device="cuda")] + [
        torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    pix = torch.arange(n, device="cuda").view(cam.height, cam.width)
    T = 32
    spent = 0.0
    for y in range(0, cam.height, T):
        row = torch.nonzero((hi[:, 1] >= y / cam.height) & (lo[:, 1] <= (y + T) / cam.height))[:, 0]
        for x in range(0, cam.width, T):
            k = row[(hi[row, 0] >= x / cam.width) & (lo[row, 0] <= (x + T) / cam.width)]
            j = pix[y:y + T, x:x + T].reshape(-1)
            spent += len(k) * len(j)
            if spent > TESTS:
                return None
            h = _closest(torch.zeros_like(d[j]), d[j], (v0[k], e1[k], e2[k]))
            out[0][j] = torch.where(h[0] >= 0, k[h[0].clamp(min=0)], -1) if len(k) else h[0]
            for a in (1, 2, 3):
                out[a][j] = h[a]
    return out


def _tuv(h, order=None):
    x = torch.stack(h[1:], 1)
    return x if order is None else x[order]


def _unit(x):
    return x / x.norm(dim=1, keepdim=True)


def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _reflect(d, n):
    return d - 2.0 * _dot(d, n) * n


def _shade(o, d, h, S, depth, budget):
    """Colours of rays o, d with hits h: the reference's materials, one recursion a level."""
    out = _t64(BACKGROUND).expand(len(o), 3).clone()
    at = torch.nonzero(h[0] >= 0)[:, 0]
    if not len(at):
        return out
    o, d, tri, t = o[at], d[at], h[0][at], h[1][at][:, None]
    b = torch.stack([1.0 - h[2][at] - h[3][at], h[2][at], h[3][at]], 1)
    f = S["idx"][tri]
    n = _unit((S["nrm"][f] * b[:, :, None]).sum(1))
    vcol = (S["colors"][f] * b[:, :, None]).sum(1)
    p = o + d * t
    hp = p + n * EPS
    mat = S["mat"][tri]
    col = torch.zeros_like(p)
    front = _dot(n, d)[:, 0] <= 0
    spec = _unit(_reflect(d, n))
    seen = []
    for pos, _, shadows in LIGHTS:
        L = _t64(pos) - hp
        lit = front & (_dot(n, L)[:, 0] > 0)
        if shadows:
            q = torch.nonzero(lit & (mat < 2))[:, 0]
            budget[0] -= len(q) * len(S["tri"][0])
            if budget[0] < 0:
                return None
            lit[q] = _closest(hp[q], L[q], S["tri"], hi=1.0)[0] < 0
        seen.append((lit, _unit(L)))
    for m, (_, amb, diffuse, power, reflexion, index, opacity) in enumerate(MATERIALS):
        q = torch.nonzero(mat == m)[:, 0]
        if not len(q):
            continue
        c = vcol[q] if m in (0, 2) else _t64(diffuse).expand(len(q), 3)
        if m >= 2:
            col[q] = (amb + (c - amb) * -_dot(n[q], _unit(d[q]))) * c
            continue
        dif, spc = torch.zeros_like(c), torch.zeros_like(c)
        for (lit, L), (_, power_of, _) in zip(seen, LIGHTS):
            on = lit[q][:, None].double()
            dif += on * _dot(n[q], L[q]) * _t64(power_of)
            spc += on * _dot(spec[q], L[q]).clamp(min=0) ** power * _t64(power_of)
        col[q] = c * (amb + dif) + spc if m == 0 else c * dif + amb + spc
        if depth == 0:
            continue
        nxt = []
        if reflexion > 0:
            nxt.append((q, _reflect(d[q], n[q]), reflexion))
        if opacity < 1:
            sgn = torch.where(front[q][:, None], 1.0, -1.0).double()
            nn, dd = n[q] * sgn, _unit(d[q])
            ratio = torch.where(front[q][:, None], 1.0 / index, index).double()
            cos = -_dot(nn, dd)
            cos2 = 1.0 - ratio * ratio * (1.0 - cos * cos)
            g = torch.nonzero(cos2[:, 0] > 0)[:, 0]
            r = dd * ratio + nn * (ratio * cos - cos2.clamp(min=0).sqrt())
            nxt.append((q[g], r[g], 1.0 - opacity))
        for at2, r, coef in nxt:
            budget[0] -= len(at2) * len(S["tri"][0])
            if budget[0] < 0:
                return None
            c2 = _shade(p[at2], r, _closest(p[at2], r, S["tri"]), S, depth - 1, budget)
            if c2 is None:
                return None
            col[at2] += coef * c2
    out[at] = col
    return out


def exact(case, seed):
    rng, kind = _rng(case, seed), case["kind"]
    if kind in ("frame", "frame_host"):
        if kind == "frame_host" or case["mesh"] == "sphere":
            verts, idx, nrm = scenes.sphere_mesh(case["lat"], case["lon"])
            verts = _deformed(verts, nrm, float(np.float32(rng.uniform(0.0, 6.0))))
            cam = _camera("sphere", case["width"], case["height"])
        else:
            verts, idx = _mesh(case, rng)
            cam = _camera("plane", case["width"], case["height"])
        h = _camera_hits(cam, _tri64(verts, idx))
        return None if h is None else {"id": None, "tuv": _tuv(h, _pixel_order(cam, case["order"])), "occluded": None}
    if kind == "diffuse":
        int(rng.integers(1 << 62))
        s = scenes.skewed_density(int(rng.integers(1 << 31)), case["tris"])
        cam = _camera("skewed", case["width"], case["height"])
        h = _camera_hits(cam, _tri64(s.verts, s.idx))
        if h is None:
            return None
        return {"primary": {"id": None, "tuv": _tuv(h, _pixel_order(cam, case["order"]))},
                "secondary": {"id": None, "tuv": None}, "rays": None}
    if kind == "build":
        verts, idx = _build_mesh(case, seed)
        return {"offsets": None, "ids": None, "records": torch.stack(_tri64(verts, idx), 1)}
    if kind in ("rays", "rays_host"):
        if case["mode"] == "any" or case["rays"] * case["tris"] > TESTS:
            return None
        s = _plane(rng, case["tris"])
        r = _random_rays(rng, case["rays"], s.verts.min(axis=0), s.verts.max(axis=0), False).double()
        h = _closest(r[:, :3].contiguous(), r[:, 4:7].contiguous(), _tri64(s.verts, s.idx))
        return {"id": None, "tuv": _tuv(h) if kind == "rays" else _tuv(h).cpu().numpy()}
    if kind == "batch":
        items = _batch_inputs(case, rng)
        if sum(len(r) * s.ntris for s, r, _ in items) > TESTS:
            return None
        got = [_tuv(_closest(r[:, :3].double(), r[:, 4:7].double(), _tri64(s.verts, s.idx))) for s, r, _ in items]
        return {"id": None, "tuv": torch.cat(got), "occluded": None}
    if kind == "instances":
        meshes, placed, cam = _instance_inputs(case, rng)
        parts = []
        for m, _, inv in placed:
            A = np.linalg.inv(np.concatenate([inv.astype(np.float64), [[0, 0, 0, 1]]]))
            parts.append(_tri64(meshes[m][0].astype(np.float64) @ A[:3, :3].T + A[:3, 3], meshes[m][1]))
        h = _camera_hits(cam, tuple(torch.cat(x) for x in zip(*parts)))
        return None if h is None else {"id": None, "tuv": _tuv(h), "instance": None}
    sc, nrm, colors, mat, cam = _render_inputs(case, rng)
    S = {"idx": torch.from_numpy(sc.idx.astype(np.int64)).cuda(), "nrm": _t64(nrm), "colors": _t64(colors),
         "mat": torch.from_numpy(mat.astype(np.int64)).cuda(), "tri": _tri64(sc.verts, sc.idx)}
    h = _camera_hits(cam, S["tri"])
    if h is None:
        return None
    o, d = _camera64(cam)
    rgb = _shade(o, d, h, S, case["depth"], [TESTS])
    return None if rgb is None else {"rgb": rgb, "rays": None}
