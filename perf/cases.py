"""The performance cases of the path tracer: what a user's program has it do, through the package's public classes.

Frames (Renderer), ray queries on device buffers (Accel, plain and precision form), two-level scenes (Batch: loading,
per-frame TLAS rebuilds, tracing) and the request loop (Server). The scenes are the box field of the benchmark in this
package (9,750 boxes = 117,002 triangles; 1,024 boxes = 12,290), drawn here with numpy from the seed, and its sphere
grid. Ray queries end at a finite tmax, beyond the scene: a miss reports t = tmax.
"""
import importlib
import math

import numpy as np
import torch

cwp = importlib.import_module("cuda-wavefront-pathtracer_b200")

HALF, EDGE_LO, EDGE_HI = 20.0, 0.2, 3.0                       # box field: ground half size, box edges
CAM_POS, CAM_TARGET, CAM_UP, HFOV = (0.0, -34.0, 22.0), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 45.0
SUN_TO, SUN_E, SUN_DEG, SKY, ALBEDO = (0.608749, -0.42625, 0.669131), 3.0, 0.526, (0.30, 0.38, 0.50), 0.7
EPS_SCALE, TMAX, BOUNCES = 1e-4, 100.0, 4
RAYS_PER_PATH = 3.7                                           # closest + shadow rays of a depth-4 path over the box field


# ---------------- the cases ----------------
def listed():
    return [
        # the benchmark's frame: one wavefront pass of 256 samples per pixel over the compressed wide BVH
        dict(name="frame_512_256spp", kind="frame", boxes=9750, layout=8, w=512, h=512, spp=256, batch=256),
        # the small configuration of the same benchmark: a thumbnail or a test render
        dict(name="frame_256_16spp", kind="frame", boxes=1024, layout=8, w=256, h=256, spp=16, batch=16),
        # a viewer that refines its image: one sample per pixel at a time, tone-mapped for display after each
        dict(name="progressive_720p", kind="progressive", boxes=9750, layout=8, w=1280, h=720, steps=4),
        # the reference's synthetic preset (sphere grid, BVH2) at an image size that is no whole number of tiles
        dict(name="frame_bvh2_spheres", kind="frame", boxes=0, layout=2, w=500, h=333, spp=16, batch=16),
        # a large batch of incoherent rays, closest hits: light baking, lidar, an external integrator's bounce
        dict(name="rays_closest_4m", kind="closest", boxes=9750, n=1 << 22),
        # a ragged batch of occlusion rays of limited reach: ambient occlusion, visibility
        dict(name="rays_any_1m", kind="any", boxes=9750, n=1_000_003),
        # a few rays, where the call's latency is what counts: picking, collision probes
        dict(name="rays_closest_2k", kind="closest", boxes=9750, n=2_000),
        # the precision form (no hit lost), closest and any
        dict(name="rays_precise_1m", kind="precise", boxes=1024, n=1 << 20),
        # many two-level scenes traced in one launch over a scene-tagged queue, closest and any
        dict(name="scenes_trace_1m", kind="scenes", scenes=8, meshes=16, tris=20_000, instances=256, n=1 << 20),
        # an animated frame: every scene's instances replaced, their TLAS rebuilt, a first set of rays traced
        dict(name="scenes_animate", kind="animate", scenes=8, meshes=8, tris=6_000, instances=1024, n=1 << 16),
        # loading: meshes to device BVHs, scenes over them, a first set of rays
        dict(name="scenes_load", kind="load", scenes=4, meshes=12, tris=40_000, instances=64, n=1 << 16),
        # the request loop: small renders of animated instanced scenes with physically based materials, served together
        dict(name="serve_small_requests", kind="serve", scenes=4, meshes=8, tris=6_000, instances=64, requests=12, res=192, spp=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "progressive", "closest", "closest", "any", "precise", "scenes", "animate", "load", "serve"])
    if kind == "frame":
        batch = rng.choice([1, 4, 16, 64])
        layout = rng.choice([8, 8, 2])
        return dict(kind=kind, boxes=_log_int(rng, 300, 9750) if layout == 8 else rng.choice([0, _log_int(rng, 300, 9750)]), layout=layout,
                    w=_log_int(rng, 64, 640), h=_log_int(rng, 64, 480), spp=batch * rng.choice([1, 2]), batch=batch)
    if kind == "progressive":
        return dict(kind=kind, boxes=_log_int(rng, 300, 9750), layout=8, w=_log_int(rng, 96, 1920), h=_log_int(rng, 96, 1080), steps=rng.randint(2, 6))
    if kind in ("closest", "any"):
        return dict(kind=kind, boxes=_log_int(rng, 300, 9750), n=_log_int(rng, 500, 1 << 22))
    if kind == "precise":
        return dict(kind=kind, boxes=_log_int(rng, 300, 4000), n=_log_int(rng, 1000, 1 << 20))
    if kind == "serve":
        return dict(kind=kind, scenes=rng.randint(2, 5), meshes=rng.randint(4, 10), tris=_log_int(rng, 1000, 12_000), instances=_log_int(rng, 8, 200),
                    requests=rng.randint(2, 16), res=rng.choice([64, 101, 128, 192, 256]), spp=rng.choice([1, 2, 4]))
    scenes = rng.randint(2, 12)
    return dict(kind=kind, scenes=scenes, meshes=rng.randint(3, 16), tris=_log_int(rng, 1000, 40_000),
                instances=_log_int(rng, 1, 1500 if kind == "animate" else 250), n=_log_int(rng, 1000, 1 << 20 if kind == "scenes" else 1 << 16))


# ---------------- scenes ----------------
QUADS = ((0, 4, 6, 2), (1, 3, 7, 5), (0, 1, 5, 4), (2, 6, 7, 3), (0, 2, 3, 1), (4, 5, 7, 6))


def box_field(n_boxes, rng):
    """(verts float32 [., 3], faces int32 [., 3]): boxes of log-uniform edges, turned about z, standing on a square ground"""
    c = rng.uniform(-HALF, HALF, (n_boxes, 2))
    e = np.exp(rng.uniform(math.log(EDGE_LO), math.log(EDGE_HI), (n_boxes, 3)))
    th = rng.uniform(0, 2 * math.pi, n_boxes)
    k = np.arange(8)
    lx, ly, lz = np.where(k & 1, 0.5, -0.5) * e[:, :1], np.where(k & 4, 0.5, -0.5) * e[:, 1:2], np.where(k & 2, 1.0, 0.0) * e[:, 2:]
    cs, sn = np.cos(th)[:, None], np.sin(th)[:, None]
    v = np.stack([c[:, :1] + lx * cs - ly * sn, c[:, 1:] + lx * sn + ly * cs, lz], -1).reshape(-1, 3)
    f = np.array([t for q in QUADS for t in ((q[0], q[1], q[2]), (q[0], q[2], q[3]))], np.int64)
    ground = np.array([[-HALF, -HALF, 0], [HALF, -HALF, 0], [HALF, HALF, 0], [-HALF, HALF, 0]])
    verts = np.concatenate([ground, v]).astype(np.float32)
    faces = np.concatenate([np.array([[0, 1, 2], [0, 2, 3]]), (4 + 8 * np.arange(n_boxes)[:, None, None] + f[None]).reshape(-1, 3)]).astype(np.int32)
    return verts, faces


def field_of(case, seed):
    return box_field(case["boxes"], np.random.default_rng([seed, 1]))


def extent_of(verts):
    return float(np.max(verts.max(0) - verts.min(0)))


def rays_of(case, seed, dev):
    """origins over the box field, directions uniform on the sphere; occlusion rays reach 8 units, the others TMAX"""
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 11)
    n = case["n"]
    o, d = torch.zeros(n, 4, device=dev), torch.empty(n, 4, device=dev)
    u = torch.rand(n, 3, generator=g, device=dev)
    o[:, 0], o[:, 1], o[:, 2] = (u[:, 0] - 0.5) * 36.0, (u[:, 1] - 0.5) * 36.0, 1.5 + 4.5 * u[:, 2]
    v = torch.randn(n, 3, generator=g, device=dev)
    d[:, :3] = v / v.norm(dim=1, keepdim=True).clamp_min(1e-12)
    d[:, 3] = 8.0 if case["kind"] == "any" else TMAX
    return o, d


def camera(case, seed):
    """pinhole camera of the benchmark, for the sphere grid turned about the scene by the seed"""
    if case["boxes"]:
        return CAM_POS, CAM_TARGET
    a = 0.37 * (seed % 17)
    return (20.0 * math.sin(a), -20.0 * math.cos(a), 8.0), (0.0, 0.0, 1.0)


def two_level(case, seed):
    """meshes [(verts, faces)], transforms [n, 12], mesh of each instance, first instance of each scene"""
    rng = np.random.default_rng([seed, 2])
    meshes = [box_field(max(1, int((case["tris"] * rng.uniform(0.25, 1.0) - 2) / 12)), rng) for _ in range(case["meshes"])]
    xf, of, first = [], [], [0]
    for s in range(case["scenes"]):
        ni = max(1, int(case["instances"] * rng.uniform(0.5, 1.5)))
        half = HALF * max(1.0, ni ** (1.0 / 3.0))
        ax = rng.normal(size=(ni, 3)); ax /= np.linalg.norm(ax, axis=1, keepdims=True)
        ang = rng.uniform(0, 2 * math.pi, ni); c, sn = np.cos(ang)[:, None, None], np.sin(ang)[:, None, None]
        cross = np.zeros((ni, 3, 3)); cross[:, 0, 1], cross[:, 0, 2], cross[:, 1, 2] = -ax[:, 2], ax[:, 1], -ax[:, 0]
        cross -= cross.transpose(0, 2, 1)
        rot = c * np.eye(3) + sn * cross + (1 - c) * ax[:, :, None] * ax[:, None, :]
        xf.append(np.concatenate([rot, rng.uniform(-half, half, (ni, 3, 1))], 2).reshape(ni, 12))
        of.append(rng.integers(0, case["meshes"], ni)); first.append(first[-1] + ni)
    return meshes, np.concatenate(xf).astype(np.float32), np.concatenate(of).astype(np.int32), np.array(first, np.int32)


def scene_rays(case, seed, first, dev):
    """rays of all scenes in one queue, scene by scene: origins uniform in the scene's cube, uniform directions"""
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 13)
    n, ns = case["n"], case["scenes"]
    sc = torch.div(torch.arange(n, device=dev) * ns, n, rounding_mode="floor").to(torch.int32)
    half = torch.tensor([HALF * max(1.0, (first[s + 1] - first[s]) ** (1.0 / 3.0)) for s in range(ns)], device=dev, dtype=torch.float32)
    o, d = torch.zeros(n, 4, device=dev), torch.empty(n, 4, device=dev)
    o[:, :3] = (2 * torch.rand(n, 3, generator=g, device=dev) - 1) * half[sc.long()][:, None]
    v = torch.randn(n, 3, generator=g, device=dev)
    d[:, :3] = v / v.norm(dim=1, keepdim=True).clamp_min(1e-12)
    d[:, 3] = 2000.0
    return o, d, sc


def with_layers(meshes):
    """meshes as the server takes them: material ids per face (ground 0, boxes 1..7)"""
    return [(v, f, np.where(np.arange(len(f)) < 2, 0, ((np.arange(len(f)) - 2) // 12) % 7 + 1).astype(np.int32), None) for v, f in meshes]


def serving(case, seed):
    meshes, _, _, _ = two_level(dict(case, scenes=1, instances=1), seed)
    rng = np.random.default_rng([seed, 3])
    mats = np.zeros((8 * len(meshes), 16), np.float32)
    mats[:, 0:3] = rng.uniform(0.2, 0.9, (len(mats), 3)); mats[:, 4:7] = 1.0; mats[:, 7] = rng.uniform(0.05, 1.0, len(mats)); mats[:, 11] = 1.5; mats[:, 12] = 1.0
    kind = rng.random(len(mats)); mats[kind < 0.1, 13] = 1.0; mats[kind > 0.75, 3] = 1.0        # glass, metal
    descs, first, reqs = [], [0], []
    halves = []
    for s in range(case["scenes"]):
        ni = max(1, int(case["instances"] * rng.uniform(0.5, 1.5)))
        half = HALF * max(1.0, ni ** (1.0 / 3.0)); halves.append(half)
        for _ in range(ni):
            d = cwp.InstanceDesc(); d.mesh = int(rng.integers(len(meshes)))
            d.translate[:] = tuple(rng.uniform(-half, half, 3)); d.translate_per_frame[:] = tuple(rng.normal(0, 0.2, 3))
            ax = rng.normal(size=3); d.axis[:] = tuple(ax / np.linalg.norm(ax))
            d.angle_deg, d.angle_deg_per_frame = float(rng.uniform(0, 360)), float(rng.uniform(-2, 2))
            d.scale[:] = (1.0, 1.0, 1.0); d.scale_per_frame[:] = (0.0, 0.0, 0.0)
            descs.append(d)
        first.append(len(descs))
    for i in range(case["requests"]):
        s = int(rng.integers(case["scenes"])); ext = 2 * (halves[s] + 30)
        th, el = rng.uniform(0, 2 * math.pi), rng.uniform(0.3, 1.2)
        pos = 0.7 * ext * np.array([math.cos(th) * math.cos(el), math.sin(th) * math.cos(el), math.sin(el)])
        w = max(16, int(case["res"] * (0.6 + 0.8 * (i % 5) / 4))); h = max(16, int(w * (0.5 + 0.5 * (i % 3) / 2)))
        reqs.append(cwp.make_request(s, cwp.camera_look_at(tuple(pos), (0, 0, 0), CAM_UP, HFOV, w, h), case["spp"], frame=int(rng.integers(30)), max_depth=8,
                                     seed=int(rng.integers(1 << 30)), eps=1e-4 * ext))
    return with_layers(meshes), mats, np.arange(0, 8 * len(meshes), 8).astype(np.int32), (cwp.InstanceDesc * len(descs))(*descs), np.array(first, np.int32), reqs


# ---------------- what a program has in hand ----------------
def frame_params(case, seed, extent):
    p = cwp.params_defaults()
    pos, target = camera(case, seed)
    p.cam = cwp.camera_look_at(pos, target, CAM_UP, HFOV, case["w"], case["h"])
    p.sun_to[:] = SUN_TO; p.sun_e[:] = (SUN_E,) * 3; p.sky[:] = SKY
    p.max_b, p.seed, p.filter_bh, p.near_clip, p.has_n = BOUNCES, 1000 + seed, 0, 0.0, 0
    return cwp.params_finish(p, SUN_DEG, EPS_SCALE, extent)


class AccumBuffer:
    """the renderer's accumulation buffer, for torch.as_tensor without a copy; a tensor made from it keeps the renderer alive"""

    def __init__(self, renderer, shape):
        self.renderer = renderer
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(int(renderer.accum_device()), False), version=3)


def prepare(case, seed):
    k, dev = case["kind"], torch.device("cuda")
    s = dict(case=case)
    if k in ("frame", "progressive"):
        mesh = cwp.Mesh.from_arrays(*field_of(case, seed)) if case["boxes"] else cwp.Mesh.sphere_grid(2)
        bvh = cwp.Bvh(mesh, variant=case["layout"], bins=32 if case["layout"] == 8 else 16)
        bvh.albedo = np.full((max(1, len(bvh.albedo)), 3), ALBEDO, np.float32)
        r = cwp.Renderer()
        p = frame_params(case, seed, extent_of(mesh.arrays()[0]))
        r.init(p, bvh, variant=case["layout"], batch=case.get("batch", 1), bounces=BOUNCES)
        s.update(r=r, accum=torch.as_tensor(AccumBuffer(r, (case["h"], case["w"], 4)), device="cuda"))
        if k == "progressive":
            s.update(rgba=torch.empty(case["h"], case["w"], 4, dtype=torch.uint8, device=dev))
    elif k in ("closest", "any", "precise"):
        bvh = cwp.Bvh(cwp.Mesh.from_arrays(*field_of(case, seed)), variant=8, bins=32)
        bvh.albedo = np.full((1, 3), ALBEDO, np.float32)
        acc = cwp.Accel(bvh)
        if k == "precise":
            acc.set_precision(1)
        o, d = rays_of(case, seed, dev)
        s.update(acc=acc, o=o, d=d, hits=torch.empty(case["n"], 4, device=dev), occ=torch.empty(case["n"], dtype=torch.int32, device=dev))
    elif k == "serve":
        meshes, mats, base, descs, first, reqs = serving(case, seed)
        batch = cwp.Batch(meshes, widths=1 << 8)
        srv = cwp.Server(batch, mats, base, max_paths=1 << 21)
        srv.set_scenes(descs, first)
        s.update(batch=batch, srv=srv, reqs=reqs)
    else:
        meshes, xf, of, first = two_level(case, seed)
        o, d, sc = scene_rays(case, seed, first, dev)
        s.update(meshes=[(v, f, None, None) for v, f in meshes], inst=cwp.instances(xf, of), first=first, o=o, d=d, sc=sc,
                 hits=torch.empty(case["n"], 4, device=dev), who=torch.empty(case["n"], dtype=torch.int32, device=dev),
                 occ=torch.empty(case["n"], dtype=torch.int32, device=dev))
        if k != "load":
            s["batch"] = cwp.Batch(s["meshes"], widths=1 << 8)
            if k == "scenes":
                s["batch"].set_scenes(s["inst"], first)
    return s


# ---------------- one pass ----------------
def hit_views(hits):
    return {"t": hits[:, 0], "uv": hits[:, 1:3], "tri": hits.view(torch.int32)[:, 3]}


def run(s):
    case = s["case"]
    k, stream = case["kind"], torch.cuda.current_stream().cuda_stream
    if k == "frame":
        st = s["r"].render(case["spp"])
        return {"accum": s["accum"], "rays": st.rays, "shadow": st.shadow_rays}
    if k == "progressive":
        for i in range(case["steps"]):
            s["r"].render(1, s_base=i, clear=i == 0)
            cwp.display(s["r"].accum_device(), s["rgba"].data_ptr(), case["w"] * case["h"], i + 1, stream=stream)
            torch.cuda.current_stream().synchronize()   # the renderer has a stream of its own: shown before the sums change
        return {"accum": s["accum"], "rgba": s["rgba"]}
    if k in ("closest", "any", "precise"):
        o, d, n = s["o"].data_ptr(), s["d"].data_ptr(), case["n"]
        out = {}
        if k != "any":
            s["acc"].trace_closest(o, d, s["hits"].data_ptr(), n, stream); out.update(hit_views(s["hits"]))
        if k != "closest":
            s["acc"].trace_any(o, d, s["occ"].data_ptr(), n, stream); out["occluder"] = s["occ"]
        return out
    if k == "serve":
        ids = [s["srv"].submit(r) for r in s["reqs"]]
        done = 0
        while done < len(ids):
            s["srv"].step()
            done += len(s["srv"].poll())
        return [s["srv"].result(i, r.cam.w, r.cam.h)[0] for i, r in zip(ids, s["reqs"])]
    batch = cwp.Batch(s["meshes"], widths=1 << 8) if k == "load" else s["batch"]
    if k != "scenes":
        batch.set_scenes(s["inst"], s["first"])
    args = s["o"].data_ptr(), s["d"].data_ptr(), s["sc"].data_ptr()
    batch.trace(*args, s["hits"].data_ptr(), s["who"].data_ptr(), case["n"], stream=stream)
    out = dict(hit_views(s["hits"]), instance=s["who"])
    if k == "scenes":
        batch.trace(*args, None, s["occ"].data_ptr(), case["n"], any_hit=True, stream=stream); out["occluder"] = s["occ"]
    if k == "load":
        torch.cuda.current_stream().synchronize()   # the batch goes away with this call
    return out


# ---------------- what a pass cannot do without ----------------
def work(case):
    """Rays read and results written once, the scene (32 B of node and 48 B of triangle per triangle) read once. Flops: each
    ray descends a tree of eight-child nodes once (8 boxes of 18 flops a level) and tests two triangles (40 flops each)."""
    k = case["kind"]
    ray = lambda tris: 144 * max(1, math.ceil(math.log(max(tris, 8) / 2, 8))) + 80  # noqa: E731
    if k in ("frame", "progressive"):
        tris = 12 * case["boxes"] + 2 if case["boxes"] else 238_400
        px, spp = case["w"] * case["h"], case.get("spp", case.get("steps"))
        return {"bytes": 80 * tris + px * 16 + (px * 4 * spp if k == "progressive" else 0), "flops": px * spp * RAYS_PER_PATH * ray(tris)}
    if k in ("closest", "any", "precise"):
        tris = 12 * case["boxes"] + 2
        both = {"closest": (48, 1), "any": (36, 1), "precise": (52, 2)}[k]
        return {"bytes": 80 * tris + case["n"] * both[0], "flops": case["n"] * both[1] * ray(tris)}
    tris, inst = case["meshes"] * case["tris"] * 0.625, case["scenes"] * case["instances"]
    if k == "serve":
        px = case["requests"] * case["res"] ** 2 * 0.75
        return {"bytes": 80 * tris + px * 16, "flops": px * case["spp"] * 6 * (ray(tris) + ray(inst) + 500)}
    passes = 2 if k == "scenes" else 1
    once = {"scenes": 80 * tris, "animate": 80 * tris + inst * (112 + 64), "load": tris * (18 + 12 + 80) + inst * (112 + 64)}[k]
    return {"bytes": once + case["n"] * (36 + 20 + 4 * (passes - 1)), "flops": case["n"] * passes * (ray(tris / case["meshes"]) + ray(inst / case["scenes"]))}


def tolerance(case):
    """Ray queries: hit distances and barycentrics are 32-bit arithmetic of a few operations per ray (against exact(): 1e-8 and
    2e-6), and of two triangles that share an edge either may be the one hit. Images: the samples of a pixel are summed by
    atomics in any order (two runs differ by 4e-8; a whole pass in another order some times that)."""
    k = case["kind"]
    if k in ("frame", "progressive"):
        return {"rel": 1e-5, "differ": 1e-3}      # differ: 8-bit values that the order of a sum tips over
    if k == "serve":
        return {"rel": 1e-5}
    return {"rel": 1e-5, "differ": 1e-5}


# ---------------- the same in 64 bits ----------------
PAIRS = 4e10                                       # ray-triangle pairs that take some seconds here
CHUNK = 1 << 27


def _cross(a, b):
    return torch.linalg.cross(a, b)


class Soup:
    """Brute-force closest and any hits in 64 bits. A ray's edge functions are products of its Pluecker coordinates with the
    triangle's, so a block of rays against all triangles is four matrix products."""

    def __init__(self, verts, faces, dev):
        v = torch.from_numpy(verts.astype(np.float64)).to(dev)[torch.from_numpy(faces.astype(np.int64)).to(dev)]
        self.v0, self.e1, self.e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        self.n = _cross(self.e1, self.e2)
        rows = [(self.v0 + self.e2, self.v0), (self.v0, self.v0 + self.e1)]      # the edges opposite to v1 (u) and v2 (v)
        self.pl = [torch.cat([_cross(a, b), b - a], 1).T.contiguous() for a, b in rows]
        self.plane = torch.cat([-self.n, (self.n * self.v0).sum(1, keepdim=True)], 1).T.contiguous()
        self.count = len(faces)

    def hits(self, o, d, tmin, tmax):
        """(t, u, v, triangle or -1) of each ray in (tmin, tmax)"""
        out = []
        step = max(1, CHUNK // self.count)
        for a in range(0, len(o), step):
            O, D = o[a:a + step], d[a:a + step]
            inv = 1.0 / (D @ self.n.T)
            t = torch.cat([O, torch.ones_like(O[:, :1])], 1) @ self.plane
            t.mul_(inv)
            ray = torch.cat([D, _cross(O, D)], 1)
            u = (ray @ self.pl[0]).mul_(inv); v = (ray @ self.pl[1]).mul_(inv)
            lim = tmax if isinstance(tmax, float) else tmax[a:a + step, None]
            ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > tmin) & (t < lim)
            t.masked_fill_(~ok, math.inf)
            best, tri = t.min(1)
            miss = torch.isinf(best)
            col = tri[:, None]
            out.append((best, u.gather(1, col)[:, 0].masked_fill(miss, 0.0), v.gather(1, col)[:, 0].masked_fill(miss, 0.0), tri.masked_fill(miss, -1)))
        return [torch.cat(x) for x in zip(*out)]


def _mix(x):
    x = x ^ (x >> 16); x = (x * 0x7FEB352D) & 0xFFFFFFFF
    x = x ^ (x >> 15); x = (x * 0x846CA68B) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _sample(pix, smp, depth, dim, seed):
    """the sample streams of the framework: a hash of (pixel, sample, depth, dimension, seed) in [0, 1)"""
    k = _mix(torch.full_like(pix, (((depth * 8 + dim) * 0xC2B2AE3D) & 0xFFFFFFFF) ^ seed))
    k = _mix(((smp * 0x85EBCA77) & 0xFFFFFFFF) ^ k)
    return (_mix(((pix * 0x9E3779B1) & 0xFFFFFFFF) ^ k) >> 8).double() / 16777216.0


def _frame_of(n):
    s = torch.where(n[:, 2] >= 0, 1.0, -1.0).double()
    a = -1.0 / (s + n[:, 2]); c = n[:, 0] * n[:, 1] * a
    return torch.stack([1 + s * n[:, 0] ** 2 * a, s * c, -s * n[:, 0]], 1), torch.stack([c, s + n[:, 1] ** 2 * a, -n[:, 1]], 1)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def exact_frame(case, seed, spp):
    """the diffuse path tracer: box-filtered camera rays, sun and constant sky, next-event estimation of the sun, cosine bounces"""
    dev = torch.device("cuda")
    verts, faces = field_of(case, seed)
    soup, w, h = Soup(verts, faces, dev), case["w"], case["h"]
    vec = lambda x: torch.tensor(x, dtype=torch.float64, device=dev)  # noqa: E731
    pos, target = (vec(x) for x in camera(case, seed))
    az = _unit(pos - target); ax = _unit(_cross(vec(CAM_UP), az)); ay = _cross(az, ax)
    focal = 0.5 * w / math.tan(math.radians(HFOV) / 2)
    sun, cos_max, eps, rs = _unit(vec(SUN_TO)), math.cos(math.radians(SUN_DEG) / 2), EPS_SCALE * extent_of(verts), 1000 + seed
    i = torch.arange(w * h * spp, device=dev)
    pix, smp = i % (w * h), torch.div(i, w * h, rounding_mode="floor")
    dx = (pix % w + _sample(pix, smp, 0, 0, rs) - 0.5 * w) / focal
    dy = -(torch.div(pix, w, rounding_mode="floor") + _sample(pix, smp, 0, 1, rs) - 0.5 * h) / focal
    d = _unit(ax * dx[:, None] + ay * dy[:, None] - az); o = pos.expand_as(d)
    T = torch.ones_like(d); image = torch.zeros(w * h, 3, dtype=torch.float64, device=dev)
    normal = _unit(soup.n)
    st, sb = _frame_of(sun[None])
    rays = shadow = 0
    for depth in range(BOUNCES + 2):
        rays += len(o)
        t, _, _, tri = soup.hits(o, d, 0.0, 1e30)
        miss = tri < 0
        image.index_add_(0, pix[miss], T[miss] * vec(SKY))
        if depth > BOUNCES:
            break
        k = ~miss
        o, d, T, pix, smp, t, ng = o[k], d[k], T[k], pix[k], smp[k], t[k], normal[tri[k]]
        ng = torch.where((ng * d).sum(1, keepdim=True) > 0, -ng, ng)
        p = o + d * t[:, None] + ng * eps
        r = [_sample(pix, smp, depth + 1, j, rs) for j in range(4)]
        cz = 1 - r[2] * (1 - cos_max); sz = (1 - cz * cz).clamp_min(0).sqrt(); ph = 2 * math.pi * r[3]
        l = _unit(sun * cz[:, None] + st * (sz * ph.cos())[:, None] + sb * (sz * ph.sin())[:, None])
        cl = (ng * l).sum(1); lit = (cl > 0).nonzero()[:, 0]
        shadow += len(lit)
        if len(lit):
            free = soup.hits(p[lit], l[lit], 0.0, 1e30)[3] < 0
            lit = lit[free]
            image.index_add_(0, pix[lit], T[lit] * (ALBEDO * SUN_E / math.pi) * cl[lit, None])
        ft, fb = _frame_of(ng); rr, ph = r[0].sqrt(), 2 * math.pi * r[1]
        d = _unit(ft * (rr * ph.cos())[:, None] + fb * (rr * ph.sin())[:, None] + ng * (1 - r[0]).clamp_min(0).sqrt()[:, None])
        k = (d * ng).sum(1) > 0
        o, d, T, pix, smp = p[k], d[k], T[k] * ALBEDO, pix[k], smp[k]
    return torch.cat([image, torch.zeros_like(image[:, :1])], 1).reshape(h, w, 4), float(rays), float(shadow)


def exact(case, seed):
    """The closest hit's distance and barycentrics by brute force, small frames by the same with the sample streams of the
    framework. None: triangle numbers (of the BVH's own order), any-hit occluders (any one may be found), 8-bit images, the two-level
    scenes (instances x triangles are too many pairs), the sphere grid and what takes too long."""
    k = case["kind"]
    tris = 12 * case.get("boxes", 0) + 2
    if k in ("frame", "progressive"):
        spp = case.get("spp", case.get("steps"))
        if not case["boxes"] or case["w"] * case["h"] * spp * RAYS_PER_PATH * tris > PAIRS * 1.5:
            return None
        image, rays, shadow = exact_frame(case, seed, spp)
        return {"accum": image, "rays": None, "shadow": None} if k == "frame" else {"accum": image, "rgba": None}
    if k not in ("closest", "precise") or case["n"] * tris > PAIRS:
        return None
    verts, faces = field_of(case, seed)
    o, d = rays_of(case, seed, torch.device("cuda"))
    t, u, v, tri = Soup(verts, faces, o.device).hits(o[:, :3].double(), d[:, :3].double(), 0.0, d[0, 3].item())
    t = torch.where(tri < 0, d[:, 3].double(), t)
    out = {"t": t, "uv": torch.stack([u, v], 1), "tri": None}
    return dict(out, occluder=None) if k == "precise" else out
