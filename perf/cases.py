"""The work whose speed this repository keeps: passes through the public entry
points (Scene, Accum, Nrc, Context.submit and the C ABI), over the sizes that
programs built on the library meet.

Kinds of case:
* frame    one frame of a scene (gbrt_render_ex), image on the host
* skinned  one animated frame: new joint matrices, skinning and refit, frame
* moving   one animated frame: new instance transforms, update, frame
* load     acceleration structures of a scene from nothing, then a frame
* trace    ray queries on device buffers, or on host arrays
* query    radiance-cache queries on device buffers
* cached   one frame through the radiance cache and one training step on it
* jobs     a batch of small frames through the job queue
"""
import ctypes
import math

import numpy as np
import torch

from rustracer_gb300 import gbrt, scenes, types as T, workloads, zoo

_ctx = None


def _context():
    """The program's one context (device, stream and scratch memory)."""
    global _ctx
    if _ctx is None:
        _ctx = gbrt.Context(0)
    return _ctx


def listed():
    return [
        # the smallest frame: a thumbnail of the 34-triangle Cornell box, all latency
        _frame("thumbnail", "cornell", 34, 64, 64, 1, 8, keep=False),
        # an interactive viewer while the camera moves: 3 samples a frame (the viewer's default) at the
        # GUI's 5 bounces, queued without waiting
        _frame("viewer", "icosphere", 20_480, 854, 480, 3, 5, queued=True),
        # a preview of every material path (textures, normal maps, alpha masks and blending, volumes, a sky
        # and a directional light) at an odd size
        _frame("materials", "zoo", 11_556, 1001, 563, 4, 8, sky=True),
        # the offline frame of the icosphere configuration: 1080p, 64 samples, depth 8, rays grouped by
        # octant as the autotuner chooses for it
        _frame("offline", "icosphere", 327_680, 1920, 1080, 64, 8, grouped=True),
        # a frame of the batched configuration: instanced tori, alpha-masked and transmissive
        _frame("instanced", "tori", 100_000, 1280, 720, 16, 8),
        # an animated frame of a 64-bone skinned mesh
        dict(name="skinned", kind="skinned", scene="tube", size=20_480, width=640, height=360, spp=2, bounces=5),
        # an animated frame of the city block: every building and sphere in a new place
        dict(name="moving", kind="moving", scene="city", size=4_000, width=960, height=540, spp=1, bounces=5),
        # opening a scene of a third of a million triangles, up to its first picture
        dict(name="load", kind="load", scene="icosphere", size=327_680, width=640, height=360, spp=1, bounces=5),
        # visibility queries of another program on its own device buffers: incoherent closest hits
        dict(name="trace", kind="trace", scene="icosphere", size=327_680, rays=1_500_001, any_hit=False, host=False),
        # radiance-cache look-ups of another program on its own device buffers
        dict(name="query", kind="query", points=1_000_003, log2_table=19),
        # a progressive frame through a radiance cache that trains as it goes
        dict(name="cached", kind="cached", scene="tori", size=20_000, width=640, height=360, spp=4, bounces=8,
             log2_table=16),
        # a batch of small frames of three scenes through the job queue
        dict(name="jobs", kind="jobs", frames=24, width=256, height=256, spp=2, bounces=8),
    ]


def _frame(name, scene, size, width, height, spp, bounces, grouped=False, queued=False, sky=False, keep=True):
    return dict(name=name, kind="frame", scene=scene, size=size, width=width, height=height, spp=spp,
                bounces=bounces, grouped=grouped, queued=queued, sky=sky, keep=keep)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _picture(rng, most):
    """Width, height and samples of a picture of at most `most` paths."""
    w = _log(rng, 33, 1920)
    h = max(17, int(w * rng.choice([9 / 16, 3 / 4, 1.0])) + rng.randrange(3) - 1)
    return dict(width=w, height=h, spp=max(1, min(_log(rng, 1, 64), most // (w * h))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "skinned", "moving", "load", "trace", "query", "cached", "jobs"])
    c = dict(kind=kind)
    if kind == "frame":
        scene, sizes = rng.choice([("cornell", [34]), ("icosphere", [1_280, 5_120, 20_480, 81_920, 327_680]),
                                   ("zoo", [11_556]), ("tori", [_log(rng, 1_000, 300_000)]), ("city", [4_000])])
        c.update(scene=scene, size=rng.choice(sizes), **_picture(rng, 1 << 24), bounces=rng.randint(1, 12),
                 grouped=rng.random() < 0.4, queued=rng.random() < 0.3, sky=scene in ("zoo", "city"),
                 keep=rng.random() < 0.7)
    elif kind == "skinned":
        c.update(scene="tube", size=_log(rng, 500, 60_000), **_picture(rng, 1 << 20), bounces=rng.randint(2, 8))
    elif kind == "moving":
        c.update(scene="city", size=_log(rng, 16, 4_000), **_picture(rng, 1 << 20), bounces=rng.randint(2, 8))
    elif kind == "load":
        scene, size = rng.choice([("icosphere", rng.choice([1_280, 20_480, 327_680])),
                                  ("tori", _log(rng, 1_000, 300_000)), ("city", _log(rng, 16, 4_000))])
        c.update(scene=scene, size=size, **_picture(rng, 1 << 20), bounces=rng.randint(2, 8))
    elif kind == "trace":
        host = rng.random() < 0.4
        scene, size = rng.choice([("icosphere", rng.choice([1_280, 20_480, 327_680])), ("zoo", 11_556),
                                  ("tori", _log(rng, 1_000, 300_000))])
        c.update(scene=scene, size=size, rays=_log(rng, 1, 200_000 if host else 4_000_000),
                 any_hit=rng.random() < 0.4, host=host)
    elif kind == "query":
        c.update(points=_log(rng, 1, 4_000_000), log2_table=rng.randint(14, 19))
    elif kind == "cached":
        c.update(scene="tori", size=_log(rng, 1_000, 100_000), **_picture(rng, 1 << 21), bounces=rng.randint(3, 10),
                 log2_table=rng.randint(14, 17))
    else:
        c.update(frames=rng.randint(1, 32), width=_log(rng, 33, 400), height=_log(rng, 33, 400),
                 spp=_log(rng, 1, 8), bounces=rng.randint(2, 8))
    return c


# --- inputs --------------------------------------------------------------------

def _scene_data(name, size, seed):
    if name == "cornell":
        return scenes.cornell()
    if name == "icosphere":  # 20 * 4^subdivision triangles
        return scenes.icosphere_scene(subdiv=int(round(math.log(size / 20, 4))), seed=seed)
    if name == "zoo":
        return zoo.material_zoo(seed=seed)
    if name == "tori":  # three meshes of about `size` triangles, two to six instances each
        return workloads.batched_scene(seed, max_tri=size, min_tri=size)[0]
    if name == "city":  # `size` instances, five eighths of them boxes
        return workloads.city_scene(seed, n_boxes=size * 5 // 8, n_spheres=size - size * 5 // 8)
    if name == "tube":  # 4 : 1 rings to segments, two triangles a quad
        segments = max(8, int(math.sqrt(size / 5)))
        return zoo.skinned_tube(rings=max(2, size // (2 * segments)), segments=segments, bones=64)
    raise ValueError(name)


def _ubo(sd, case, rng):
    """The case's frame from an eye near the scene's own."""
    eye = np.asarray(sd.camera["eye"], np.float64) + rng.uniform(-0.05, 0.05, 3)
    return sd.ubo(case["width"], case["height"], eye=tuple(eye), samples=case["spp"], bounces=case["bounces"],
                  has_sky=bool(case.get("sky")) or case["scene"] == "city")


def _pinned_image(case):
    return torch.zeros((case["height"], case["width"], 4), dtype=torch.uint8, pin_memory=True).numpy()


def _box(sd, pad=0.5):
    return workloads.world_box(sd, pad)


def _points(n, lo, hi, rng):
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = rng.uniform(lo, hi, (n, 3))
    return p


def _rays(sd, case, rng):
    """Incoherent rays like a path's later bounces: origins all over the scene, directions over the sphere."""
    lo, hi = _box(sd, 0.1)
    r = scenes.random_rays(case["rays"], seed=int(rng.integers(1 << 31)))
    r["org"] = rng.uniform(lo, hi, (case["rays"], 3))
    r["tmin"] = 1e-3
    return r


def _cache_parameters(case, rng):
    """MLP and table of a cache that has been trained: weights of the initialisation's spread, features of order 1."""
    fan = np.concatenate([np.full(64 * 32, math.sqrt(6 / 32)), np.full(gbrt.Nrc.MLP_PARAMS - 64 * 32, math.sqrt(6 / 64))])
    mlp = (rng.uniform(-1, 1, gbrt.Nrc.MLP_PARAMS) * fan).astype(np.float32)
    return mlp, rng.uniform(-0.5, 0.5, 32 << case["log2_table"]).astype(np.float32)


def prepare(case, seed):
    ctx, rng, kind = _context(), np.random.default_rng(seed), case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "query":
        s["cache"] = gbrt.Nrc(ctx, (-2.0,) * 3, (2.0,) * 3, log2_table=case["log2_table"])
        s["cache"].set_params(*_cache_parameters(case, rng))
        s["points"] = torch.from_numpy(_points(case["points"], -2.0, 2.0, rng)).cuda()
        s["out"] = torch.zeros_like(s["points"])
        return s
    if kind == "jobs":
        s["work"] = []
        sds = [scenes.cornell(), scenes.icosphere_scene(subdiv=4, seed=seed), zoo.material_zoo(seed=seed)]
        built = [gbrt.Scene(ctx, sd) for sd in sds]
        for k in range(case["frames"]):
            sd = sds[k % 3]
            ubo = _ubo(sd, dict(case, scene=""), rng)
            s["work"].append((built[k % 3], ubo, gbrt.Accum(ctx, case["width"], case["height"])))
        return s
    sd = _scene_data(case["scene"], case["size"], seed)
    s["scene"] = gbrt.Scene(ctx, sd)
    if case.get("grouped"):
        s["scene"].set_tuning(8, True)
    if kind == "trace":
        rays = _rays(sd, case, rng)
        if case["host"]:
            s["rays"] = rays
        else:
            s["rays"] = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
            s["hits"] = torch.zeros((case["rays"], 6), device="cuda")
        return s
    s["ubo"] = _ubo(sd, case, rng)
    s["accum"] = gbrt.Accum(ctx, case["width"], case["height"])
    s["image"] = _pinned_image(case) if case.get("keep", True) else None
    if kind == "skinned":
        s["skins"] = zoo.bone_matrices(sd.bones, rng.uniform(0, 6.28))
    elif kind == "moving":
        inst = sd.instances.copy()
        step = rng.uniform(-0.2, 0.2, (len(inst), 3)).astype(np.float32)
        step[0] = 0.0  # the ground stays
        inst["transform"].reshape(-1, 3, 4)[:, :, 3] += step
        s["instances"] = inst
    elif kind == "cached":
        lo, hi = _box(sd)
        s["cache"] = gbrt.Nrc(ctx, lo, hi, log2_table=case["log2_table"], learning_rate=1e-3, seed=seed)
    return s


# --- passes ----------------------------------------------------------------------

def _render(s):
    r = s["scene"].render(s["ubo"], s["accum"], out=s["image"])
    return dict(image=r["image"], rays=int(r["stats"]["rays_total"]))


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "frame":
        if case["queued"]:  # the image is complete once the device is waited for
            return dict(image=s["scene"].render(s["ubo"], s["accum"], asynchronous=True, out=s["image"])["image"])
        return _render(s)
    if kind == "skinned":
        s["scene"].skin_and_refit(s["skins"])
        return _render(s)
    if kind == "moving":
        s["scene"].update_tlas(s["instances"])
        return _render(s)
    if kind == "load":
        s["scene"].create_as()
        return _render(s)
    if kind == "trace":
        flags = 0x4 if case["any_hit"] else 0  # GBRT_RAY_TERMINATE_ON_FIRST
        if case["host"]:
            hits, _ = s["scene"].trace(s["rays"], flags)
            if case["any_hit"]:
                return dict(hit=hits["instance_id"] != 0xFFFFFFFF)
            return dict(t=hits["t"], u=hits["u"], v=hits["v"], instance=hits["instance_id"].astype(np.int64),
                        primitive=hits["primitive_id"].astype(np.int64))
        ctx.check(ctx.L.gbrt_trace_rays_device(s["scene"].h, ctypes.c_void_p(s["rays"].data_ptr()), case["rays"],
                                               flags, ctypes.c_void_p(s["hits"].data_ptr())))
        ids = s["hits"].view(torch.int32)
        if case["any_hit"]:  # which of a ray's occluders is reported is not specified
            ctx.sync()
            return dict(hit=ids[:, 3] != -1)
        return dict(t=s["hits"][:, 0], u=s["hits"][:, 1], v=s["hits"][:, 2], instance=ids[:, 3], primitive=ids[:, 4])
    if kind == "query":
        s["cache"].query_device(s["points"].data_ptr(), case["points"], s["out"].data_ptr())
        return dict(radiance=s["out"][:, :3])
    if kind == "cached":
        r = s["cache"].render(s["scene"], s["ubo"], s["accum"], image=False)
        mlp, table = s["cache"].params()
        return dict(sum=s["accum"].download()[..., :3], loss=r["loss"], mlp=mlp, table=table)
    pending = [ctx.submit(scene, ubo, accum) for scene, ubo, accum in s["work"]]
    for j in pending:
        j.wait()
    return [j.image for j in pending]


def exact(case, seed):
    if case["kind"] == "query":
        return _exact_query(case, seed)
    if case["kind"] == "trace" and not case["any_hit"]:
        return _exact_trace(case, seed)
    return None  # Monte Carlo pictures: bytes, and paths that follow their rounding


def _exact_trace(case, seed):
    """Closest hits by testing every triangle in 64 bits; None where that takes too long or an alpha test decides."""
    sd = _scene_data(case["scene"], case["size"], seed)
    if case["scene"] != "icosphere" or case["rays"] * sd.num_triangles > 4_000_000_000:
        return None
    rays = _rays(sd, case, np.random.default_rng(seed))
    vert = sd.vertices["pos"][:, :3].astype(np.float64)
    tri = np.concatenate([vert[int(p["v_offset"]) + sd.indices[int(p["i_offset"]):int(p["i_offset"]) + int(g["i_len"])]]
                          for p, g in zip(sd.prims, sd.geo_ranges)]).reshape(-1, 3, 3)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p0, p1, p2 = (torch.from_numpy(np.ascontiguousarray(tri[:, k])).to(dev) for k in range(3))
    e1, e2 = p1 - p0, p2 - p0
    found = []
    step = max(1, 20_000_000 // len(tri))
    for at in range(0, case["rays"], step):
        r = rays[at:at + step]
        o = torch.from_numpy(r["org"].astype(np.float64)).to(dev)[:, None]
        d = torch.from_numpy(r["dir"].astype(np.float64)).to(dev)[:, None]
        h = torch.linalg.cross(d.expand(-1, len(e2), -1), e2[None].expand(len(r), -1, -1))
        a = (e1 * h).sum(-1)
        f = o - p0
        q = torch.linalg.cross(f, e1[None].expand(len(r), -1, -1))
        u, v, t = (f * h).sum(-1) / a, (d * q).sum(-1) / a, (e2 * q).sum(-1) / a
        ok = (a != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 1e-3) & (t <= 1e4)
        t, k = torch.where(ok, t, math.inf).min(1, keepdim=True)
        hit = torch.isfinite(t)
        zero = torch.zeros_like(t)
        found.append(torch.cat([torch.where(hit, t, zero - 1), torch.where(hit, u.gather(1, k), zero),
                                torch.where(hit, v.gather(1, k), zero)], 1))
    found = torch.cat(found)
    return dict(t=found[:, 0], u=found[:, 1], v=found[:, 2], instance=None, primitive=None)


def _exact_query(case, seed):
    """The hash-grid encoding and the MLP in 64 bits, on the parameters as uploaded."""
    rng = np.random.default_rng(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    mlp, table = (torch.from_numpy(a).to(dev).double() for a in _cache_parameters(case, rng))
    p = torch.from_numpy(_points(case["points"], -2.0, 2.0, rng)[:, :3]).to(dev).double()
    p = ((p + 2.0) / 4.0).clamp(0.0, 1.0)
    entries = 1 << case["log2_table"]
    table = table.reshape(16, entries, 2)
    features = []
    for level in range(16):
        scale = float(np.float32(16.0 * float(np.float32(1.447)) ** level - 1.0))
        res = math.ceil(scale) + 2
        g = p * scale + 0.5
        cell = g.floor()
        w, cell = g - cell, cell.long()
        x = 0.0
        for corner in range(8):
            bit = torch.tensor([corner & 1, corner >> 1 & 1, corner >> 2], device=dev)
            c = cell + bit
            if res ** 3 <= entries:
                at = c[:, 0] + c[:, 1] * res + c[:, 2] * res * res
            else:
                at = (c[:, 0] ^ (c[:, 1] * 2654435761) ^ (c[:, 2] * 805459861)) & (entries - 1)
            x = x + torch.where(bit.bool(), w, 1.0 - w).prod(1, keepdim=True) * table[level, at]
        features.append(x)
    h, at = torch.cat(features, 1), 0
    for rows, cols in [(64, 32)] + [(64, 64)] * 4 + [(3, 64)]:
        h = h @ mlp[at:at + rows * cols].reshape(rows, cols).T
        h, at = (h.relu() if rows == 64 else h), at + rows * cols
    return dict(radiance=h)


# --- what a pass cannot do without ------------------------------------------------

def _geometry(case):
    """(bytes, world triangles) of a case's scene: vertices, indices and instances, each once."""
    size = case["size"]
    if case["scene"] == "tori":  # 12 instances on average of three meshes
        return 3 * size * (64 + 12), 12 * size
    if case["scene"] == "city":
        return 642 * 128 + 16 * 1_280 * 12 + 64 * size, size * 5 // 8 * 12 + (size - size * 5 // 8) * 1_280
    return size * (64 + 12), size


def _frame_work(case, scene_bytes, triangles):
    """A picture: the scene read once, the running sum and the image written; per path about four rays, each at
    least one box test (12 operations) a binary level and two triangle tests (60), and two shaded hits (800)."""
    pixels = case["width"] * case["height"]
    paths = pixels * case["spp"]
    per_ray = 12 * math.log2(max(2, triangles)) + 120
    return scene_bytes + pixels * 20, paths * (4 * per_ray + 1_600)


def work(case):
    kind = case["kind"]
    if kind == "query":  # position in, radiance out, the 16-bit table once; 37,248 operations of the MLP
        n = case["points"]
        return dict(bytes=n * 32 + min(n * 512, 64 << case["log2_table"]), flops=n * (37_248 + 16 * 8 * 4))
    if kind == "jobs":
        b, f = _frame_work(dict(case, scene="icosphere"), 0, 5_000)
        return dict(bytes=case["frames"] * b + 16_000 * 76, flops=case["frames"] * f)
    scene_bytes, triangles = _geometry(case)
    if kind == "trace":
        n = case["rays"]
        return dict(bytes=n * (32 + 24) + triangles * 36, flops=n * (12 * math.log2(max(2, triangles)) + 120))
    b, f = _frame_work(case, scene_bytes, triangles)
    if kind == "skinned":  # vertices read and written (128 bytes, one for two triangles); boxes of all triangles
        b, f = b + triangles * 128, f + triangles * 200
    elif kind in ("moving", "load"):  # each triangle's box and one tree over them, written once
        b, f = b + triangles * (36 + 64), f + triangles * 300
    elif kind == "cached":  # 2^16 samples: three products of the MLP and its gradients; table, moments and gradient
        table = 128 << case["log2_table"]
        b, f = b + 6 * table, f + 65_536 * 111_744
    return dict(bytes=b, flops=f)
