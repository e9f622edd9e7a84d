"""Performance cases of the path tracer: what its users have it do, through the public entry points of ptgb.

A case is a dict of plain values; its "kind" says which call it stands for:

  pick     first hit of every camera ray (object picking, id masks, depth)
  frame    one progressive frame of an interactive session: a short render and the display conversion
  render   an offline render of a whole image
  commit   a scene rebuilt after an edit (upload and BVH build), and the first hits of the new scene
  batch    many small scenes in one wavefront (data-set generation)
  guided   frames with the learned sampling guide and its online training, double sums

listed() has the sizes of this repository's benchmark, examples and tests; draw() spreads them over the same ranges.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "optix-path-tracer_gb300"))
import ptgb  # noqa: E402

REF, CONSISTENT = 0, 1


def listed():
    return [
        # picking in a small viewport: the smallest call there is, all launch and copy latency
        {"name": "pick_cornell_96", "kind": "pick", "scene": "cornell", "width": 96, "height": 64, "size": 0},
        # the interactive loop of the reference application: one frame of its Cornell box per launch, then the display
        {"name": "frame_cornell_500", "kind": "frame", "scene": "cornell", "width": 500, "height": 500, "spp": 1, "mode": REF, "size": 0},
        # the same loop at full HD on the spheres scene, without lights
        {"name": "frame_spheres_1080p", "kind": "frame", "scene": "spheres", "width": 1920, "height": 1080, "spp": 1, "mode": REF, "size": 11},
        # the same loop in a terrain viewer: triangles, HDR sky, next-event estimation with MIS
        {"name": "frame_terrain_720p", "kind": "frame", "scene": "terrain", "width": 1280, "height": 720, "spp": 1, "mode": CONSISTENT, "size": 512},
        # motion blur preview, odd image size and frame count
        {"name": "moving_637x361_5", "kind": "render", "scene": "moving", "width": 637, "height": 361, "spp": 5, "mode": REF, "size": 5},
        # every texture callable and nearly every BRDF, odd image size
        {"name": "textures_321x243_33", "kind": "render", "scene": "textures", "width": 321, "height": 243, "spp": 33, "mode": CONSISTENT, "size": 0},
        # benchmark workload: Cornell box, 64 frames
        {"name": "cornell_512_64", "kind": "render", "scene": "cornell", "width": 512, "height": 512, "spp": 64, "mode": REF, "size": 0},
        # benchmark workload: random spheres, 128 frames
        {"name": "spheres_1080p_128", "kind": "render", "scene": "spheres", "width": 1920, "height": 1080, "spp": 128, "mode": REF, "size": 11},
        # benchmark workload: 2.1 M triangles under an importance-sampled sky, one 64-frame chunk
        {"name": "terrain_1080p_64", "kind": "render", "scene": "terrain", "width": 1920, "height": 1080, "spp": 64, "mode": CONSISTENT, "size": 1024},
        # an edit of the 2.1 M-triangle scene
        {"name": "commit_terrain_1024", "kind": "commit", "scene": "terrain", "width": 640, "height": 360, "size": 1024},
        # scenes of very different sizes in one batch
        {"name": "batch_8", "kind": "batch", "scene": "terrain", "items": 8, "side": 512, "spp": 48, "mode": CONSISTENT, "size": 500},
        # the learned guide in a closed box lit through a small opening
        {"name": "guided_540p_4", "kind": "guided", "scene": "box", "width": 960, "height": 540, "spp": 4, "mode": CONSISTENT, "size": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, lo, hi):
    """A width and a height with lo..hi pixels between them, odd ones among them."""
    pixels, aspect = math.exp(rng.uniform(math.log(lo), math.log(hi))), rng.uniform(0.75, 2.4)
    w = max(1, int(math.sqrt(pixels * aspect)))
    return w, max(1, int(pixels / w))


def draw(rng):
    kind = rng.choice(["pick", "frame", "frame", "render", "render", "render", "commit", "batch", "guided"])
    if kind == "pick":
        w, h = _image(rng, 1000, 1 << 21)
        return {"kind": kind, "scene": "cornell", "width": w, "height": h, "size": 0}
    if kind == "commit":
        w, h = _image(rng, 10000, 1 << 18)
        return {"kind": kind, "scene": "terrain", "width": w, "height": h, "size": _log_int(rng, 24, 1024)}
    if kind == "batch":
        return {"kind": kind, "scene": "terrain", "items": rng.randint(2, 10), "side": rng.choice([128, 255, 256, 511, 512]),
                "spp": rng.randint(4, 48), "mode": rng.choice([REF, CONSISTENT, CONSISTENT]), "size": _log_int(rng, 24, 500)}
    if kind == "guided":
        w, h = _image(rng, 20000, 518400)
        return {"kind": kind, "scene": "box", "width": w, "height": h, "spp": rng.randint(1, 4), "mode": CONSISTENT, "size": _log_int(rng, 32, 512)}
    scene = rng.choice(["cornell", "spheres", "terrain", "moving", "textures"])
    size = {"spheres": rng.randint(2, 11), "moving": rng.randint(2, 8), "terrain": _log_int(rng, 24, 1024)}.get(scene, 0)
    w, h = _image(rng, 4000, 1920 * 1080)
    spp = rng.randint(1, 2) if kind == "frame" else max(2, min(_log_int(rng, 2, 256), (48 << 20) // (w * h)))
    mode = rng.choice([REF, CONSISTENT]) if scene != "terrain" else CONSISTENT
    return {"kind": kind, "scene": scene, "width": w, "height": h, "spp": spp, "mode": mode, "size": size}


# ------------------------------------------------------------------ scenes
def _terrain_mesh(cells, gen):
    """(cells + 1)^2 vertices over [-1, 1]^2 with six octaves of smooth noise; vertices, normals, uvs, indices and the tile (16 x 16) of each triangle."""
    n = cells + 1
    y = torch.zeros(n, n)
    for o in range(6):
        grid = torch.rand(1, 1, (4 << o) + 1, (4 << o) + 1, generator=gen) * 2 - 1
        y += 0.5 ** o * torch.nn.functional.interpolate(grid, size=(n, n), mode="bicubic", align_corners=True)[0, 0]
    y *= 0.1 / 1.97
    lin = torch.linspace(-1, 1, n)
    z, x = torch.meshgrid(lin, lin, indexing="ij")
    gz, gx = torch.gradient(y, spacing=2.0 / cells)
    nrm = torch.nn.functional.normalize(torch.stack([-gx, torch.ones_like(gx), -gz], -1), dim=-1)
    uv = torch.stack([(x + 1) / 2, (z + 1) / 2], -1)
    j, i = torch.meshgrid(torch.arange(cells), torch.arange(cells), indexing="ij")
    v0 = (j * n + i).reshape(-1)
    idx = torch.stack([v0, v0 + n, v0 + 1, v0 + 1, v0 + n, v0 + n + 1], -1).reshape(-1, 3)
    tile = ((j * 16 // cells) * 16 + i * 16 // cells).reshape(-1).repeat_interleave(2)
    verts = torch.stack([x, y, z], -1)
    return [t.numpy() for t in (verts.reshape(-1, 3), nrm.reshape(-1, 3), uv.reshape(-1, 2), idx.to(torch.int32), tile)]


def _sky(w, h, gen):
    """HDR sky with a sun lobe in a seeded direction: RGBA float, row 0 at v = 0, the zenith first."""
    lat = ((torch.arange(h) + 0.5) / h * math.pi)[:, None]
    lon = ((torch.arange(w) + 0.5) / w * 2 * math.pi)[None, :]
    d = torch.stack([(lat.sin() * lon.cos()), lat.cos().expand(h, w), lat.sin() * lon.sin()], -1)
    t = d[..., 1:2].clamp(0, 1)
    sky = (1 - t) * torch.ones(3) + t * torch.tensor([0.3, 0.5, 1.0])
    col = torch.where(d[..., 1:2] >= 0, sky, torch.tensor([0.15, 0.12, 0.1]))
    az = float(torch.rand(1, generator=gen)) * 2 * math.pi
    sun = torch.tensor([math.cos(az) * 0.8, 0.6, math.sin(az) * 0.8])
    ang = (d @ sun).clamp(-1, 1).acos()
    col = col + 5e4 * torch.exp(-0.5 * (ang / 0.03) ** 2)[..., None] * torch.tensor([1, 0.9, 0.8])
    return torch.cat([col, torch.zeros(h, w, 1)], -1).contiguous().numpy()


def _terrain(cells, width, height, seed, env):
    gen = torch.Generator().manual_seed(seed)
    verts, nrm, uv, idx, tile = _terrain_mesh(cells, gen)
    u = torch.rand(256, 7, generator=gen).tolist()
    s = ptgb.Scene()
    mats = []
    for k, r, g, b, p, q, c in u:
        col = (0.3 + 0.6 * r, 0.3 + 0.6 * g, 0.3 + 0.6 * b)
        if k < 1 / 3:
            mats.append(s.torrance_sparrow(col, 0.05 + 0.45 * p, 0.05 + 0.45 * p))
        elif k < 2 / 3:
            mats.append(s.ashikhmin_shirley(col, (0.04 + 0.2 * c,) * 3, 10 + 990 * p, 10 + 990 * q))
        else:
            mats.append(s.oren_nayar(col, 0.5 * p))
    s.mesh(verts, idx, mats[0], mat_per_tri=np.asarray(mats, np.uint32)[tile], normals=nrm, uvs=uv)
    s.miss_env(_sky(*env, gen), spherical=True)
    s.set_camera((0.0, 0.9, 1.9), (0.0, 0.0, 0.0), (0, 1, 0), 45.0, width / height, 0.0, 2.0)
    return s


def _box(cells, width, height, seed):
    """The terrain in a closed white box whose ceiling has a small square opening to the sky; the camera is inside."""
    s = _terrain(cells, width, height, seed, (1024, 512))
    wall = s.lambertian((0.7, 0.7, 0.7))
    x, y0, y1, side = 1.02, -0.2, 1.2, 0.3
    a0, b0 = 0.2, 0.1
    a1, b1 = a0 + side, b0 + side
    for k, flip in ((-x, False), (x, True)):
        s.rect(y0, y1, -x, x, k, flip, ptgb.PT_X_AXIS, wall)
        s.rect(-x, x, y0, y1, k, flip, ptgb.PT_Z_AXIS, wall)
    s.rect(-x, x, -x, x, y0, False, ptgb.PT_Y_AXIS, wall)
    for r in ((-x, a0, -x, x), (a1, x, -x, x), (a0, a1, -x, b0), (a0, a1, b1, x)):
        s.rect(*r, y1, True, ptgb.PT_Y_AXIS, wall)
    s.set_camera((0.0, 0.75, 0.98), (0.0, 0.0, -0.3), (0, 1, 0), 60.0, width / height, 0.0, 2.0)
    return s


def _cornell(width, height, seed):
    """The benchmark's Cornell box with its two boxes at seeded angles."""
    s = ptgb.cornell_c1(width, height)
    angles = np.random.RandomState(seed).uniform(-25, 25, 2)
    for k, (name, p0, p1, m, _) in [(k, it) for k, it in enumerate(s.items) if it[0] == "box"]:
        at = (130.0, 0.0, 65.0) if p1[1] < 200 else (265.0, 0.0, 295.0)
        xf = ptgb.compose([ptgb.mat_translate(at), ptgb.mat_rotate(float(angles[0 if p1[1] < 200 else 1]), ptgb.PT_Y_AXIS)])
        s.items[k] = (name, p0, p1, m, xf)
    return s


def _textures(width, height, seed):
    """The texture scene with its spheres' heights and the camera's seeded."""
    s = ptgb.texture_zoo(width, height)
    r = np.random.RandomState(seed)
    for k, it in enumerate(s.items):
        if it[0] == "sphere":
            s.items[k] = ("sphere", (it[1][0], it[1][1] + float(r.uniform(0, 0.3)), it[1][2])) + it[2:]
    s.set_camera((float(r.uniform(-0.5, 0.5)), 1.6, 4.5), (0.0, 0.3, 0.0), (0, 1, 0), 45.0, width / height, 0.05, 4.5)
    return s


def _scene(c, seed):
    kind, w, h = c["scene"], c.get("width", 1), c.get("height", 1)
    if kind == "cornell":
        return _cornell(w, h, seed % (1 << 31))
    if kind == "spheres":
        return ptgb.random_spheres(w, h, seed, c["size"])
    if kind == "moving":
        return ptgb.moving_spheres(w, h, seed, c["size"])
    if kind == "textures":
        return _textures(w, h, seed % (1 << 31))
    if kind == "box":
        return _box(c["size"], w, h, seed)
    return _terrain(c["size"], w, h, seed, (2048, 1024) if c["size"] > 600 else (1024, 512))


# ---------------------------------------------------------------- the calls
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        jobs = []
        for k in range(case["items"]):
            # triangle counts, image sides and frame counts differ from item to item
            f = 0.05 ** (((k * 5) % 8) / 8)
            side = max(16, case["side"] * (2 if k % 3 == 1 else 1) // (2 if k % 3 == 2 else 1))
            spp = max(1, case["spp"] * (1 + k % 4) // 4)
            s = _terrain(max(16, int(case["size"] * f)), side, side, seed * 64 + k, (512, 256))
            acc = torch.zeros(side, side, 4, device="cuda")
            jobs.append((ptgb.GpuRenderer(s), ptgb.GpuRenderer.params(side, side, spp, mode=case["mode"]), acc))
        return {"kind": kind, "batch": ptgb.Batch(), "jobs": [(r, p, a.data_ptr()) for r, p, a in jobs], "accs": [a for _, _, a in jobs]}
    r = ptgb.GpuRenderer(_scene(case, seed))
    st = {"kind": kind, "r": r, "w": case["width"], "h": case["height"]}
    if kind in ("pick", "commit"):
        return st
    w, h = case["width"], case["height"]
    rr = 3 if case["scene"] == "cornell" else 10
    st["params"] = r.params(w, h, case["spp"], mode=case["mode"], rr_depth=rr, guide=1 if kind == "guided" else 0)
    if kind == "guided":
        st["seed"] = seed
        st["acc"] = torch.zeros(h, w, 4, dtype=torch.float64, device="cuda")
    elif kind == "render" and case["scene"] == "cornell":
        st["acc"] = np.zeros((h, w, 4), np.float32)  # a program that writes the image to a file has it in host memory
    else:
        st["acc"] = torch.zeros(h, w, 4, device="cuda")
    if kind == "frame":
        st["rgba8"] = np.zeros((h, w, 4), np.uint8)
    return st


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].render(state["jobs"])
        return state["accs"]
    r = state["r"]
    if kind == "pick":
        return r.first_hits(state["w"], state["h"], 0)
    if kind == "commit":
        r._c(r.lib.pt_commit(r.ctx))
        return r.first_hits(state["w"], state["h"], 0)
    acc = state["acc"]
    ptr = acc if isinstance(acc, np.ndarray) else acc.data_ptr()
    if kind == "guided":
        r.guide_init(state["seed"])  # an image starts with an untrained guide
        r.render64(state["params"], ptr)
        weights, step = r.guide_state()
        return acc, weights, step
    r.render(state["params"], ptr)
    if kind == "frame":
        r._c(r.lib.pt_resolve_display(r.ctx, ptr, state["w"], state["h"], state["params"].spp - 1, state["rgba8"].ctypes.data, None))
        return acc, state["rgba8"]
    return acc


# --------------------------------------------------------------- what it takes
def work(case):
    """Bytes: the scene's geometry read once, each output written once. Operations: per ray one descent of a tree over the scene (eight boxes a
    level) and one primitive, per bounce its shading; rays per path as these scenes have them."""
    prims = {"terrain": 2 * case["size"] ** 2, "box": 2 * case["size"] ** 2, "spheres": 4 * case["size"] ** 2 + 4, "moving": 4 * case["size"] ** 2 + 4}.get(case["scene"], 16)
    rays = {"cornell": 9.0, "spheres": 2.8, "terrain": 2.1, "moving": 3.5, "textures": 4.0, "box": 12.0}[case["scene"]]
    per_ray = 8 * 12 * max(1.0, math.log(prims, 8)) + 60 + 150
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["items"]):
            side = max(16, case["side"] * (2 if k % 3 == 1 else 1) // (2 if k % 3 == 2 else 1))
            paths = side * side * max(1, case["spp"] * (1 + k % 4) // 4)
            p = 2 * max(16, int(case["size"] * 0.05 ** (((k * 5) % 8) / 8))) ** 2
            total["bytes"] += 48 * p + side * side * 16
            total["flops"] += paths * rays * per_ray
        return total
    pixels = case["width"] * case["height"]
    if case["kind"] == "pick":
        return {"bytes": 48 * prims + 12 * pixels, "flops": pixels * (per_ray - 150)}
    if case["kind"] == "commit":
        # records read, records and nodes written; the attributes and the sky go to the device
        env = 16 * (2048 * 1024 if case["size"] > 600 else 1024 * 512)
        return {"bytes": prims * (48 + 48 + 12 + 26 + 4) + env + 12 * pixels, "flops": pixels * (per_ray - 150) + 100 * prims}
    paths = pixels * case["spp"]
    out = {"frame": 16 + 4, "render": 16, "guided": 32}[case["kind"]]
    return {"bytes": 48 * prims + out * pixels, "flops": paths * rays * per_ray}


# ------------------------------------------------------------------ 64 bits
def _tea64(v0, v1):
    v0, v1 = v0.astype(np.uint32), v1.astype(np.uint32)
    s = np.uint32(0)
    with np.errstate(over="ignore"):
        for _ in range(64):
            s = np.uint32((int(s) + 0x9E3779B9) & 0xFFFFFFFF)
            v0 = v0 + (((v1 << np.uint32(4)) + np.uint32(0xA341316C)) ^ (v1 + s) ^ ((v1 >> np.uint32(5)) + np.uint32(0xC8013EA4)))
            v1 = v1 + (((v0 << np.uint32(4)) + np.uint32(0xAD90777D)) ^ (v0 + s) ^ ((v0 >> np.uint32(5)) + np.uint32(0x7E95761E)))
    return v0


def exact(case, seed):
    """Distances of the first hits in the Cornell box in 64 bits (ids have no 64-bit form). A path's colour has none: which way it goes
    hangs on comparisons of 32-bit values."""
    if case["kind"] != "pick":
        return None
    w, h = case["width"], case["height"]
    s = _cornell(w, h, seed % (1 << 31))
    y, x = np.divmod(np.arange(w * h, dtype=np.uint32), np.uint32(w))
    state = _tea64(np.arange(w * h, dtype=np.uint32), np.zeros(w * h, np.uint32))
    u = []
    for _ in range(2):
        with np.errstate(over="ignore"):
            state = state * np.uint32(1664525) + np.uint32(1013904223)
        u.append((state & np.uint32(0xFFFFFF)) / 16777216.0)
    cf, ca, up, vfov, aspect, _, focus = [np.asarray(v, np.float64) for v in s.camera[:7]]
    hh = math.tan(float(vfov) * math.pi / 360)
    cw = (cf - ca) / np.linalg.norm(cf - ca)
    cu = np.cross(up, cw)
    cu /= np.linalg.norm(cu)
    cv = np.cross(cw, cu)
    a, b = (x + u[0]) / w * 2 - 1, (y + u[1]) / h * 2 - 1
    o = cf
    d = float(focus) * (a[:, None] * hh * float(aspect) * cu + b[:, None] * hh * cv - cw)
    best = np.full(w * h, np.inf)
    for it in s.items:
        with np.errstate(divide="ignore", invalid="ignore"):
            if it[0] == "rect":
                (a0, a1, b0, b1, k), axis = it[1], it[3]
                i, j = [(1, 2), (0, 2), (0, 1)][axis]
                t = (k - o[axis]) / d[:, axis]
                p, q = o[i] + t * d[:, i], o[j] + t * d[:, j]
                ok = (p >= a0) & (p <= a1) & (q >= b0) & (q <= b1)
            else:
                m = np.asarray(it[4], np.float64).reshape(3, 4)
                inv = np.linalg.inv(m[:, :3])
                oo, dd = inv @ (o - m[:, 3]), d @ inv.T
                t0, t1 = (np.asarray(it[1], np.float64) - oo) / dd, (np.asarray(it[2], np.float64) - oo) / dd
                t, far = np.minimum(t0, t1).max(1), np.maximum(t0, t1).min(1)
                ok = t <= far
        best = np.where(ok & (t > 1e-6) & (t < best), t, best)
    return None, None, np.where(np.isinf(best), 0.0, best)
