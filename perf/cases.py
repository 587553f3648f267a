"""The work that is timed: renders, batched views, served requests, real-time frames, denoising and relighting.

Each case is what a program does with this framework through its public entry points, on the
framework's own procedural scenes (the closed box of 36 triangles and the height-field scenes), at
sizes from a thumbnail to the 1080p frame of the benchmark. `listed()` names the fixed cases,
`draw(rng)` gives others of the same ranges, `prepare` makes a case's inputs on the GPU, `run` is one
pass, `work` the bytes and operations a pass cannot do without, and `exact` the denoiser's result in
64 bits (a path-traced image has no such value: it is an estimate whose random walk depends on every
rounding).
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from photon_b200 import abi, native, workloads

BOX = 36


def _render(name, triangles, width, height, spp, depth, camera="scene", aperture=0.0, clamp=0.0):
    return {"name": name, "kind": "render", "triangles": triangles, "width": width, "height": height, "spp": spp, "depth": depth,
            "camera": camera, "aperture": aperture, "clamp": clamp}


def listed():
    return [
        # A thumbnail or a material preview: the smallest call, launches and latency.
        _render("box_64x64_4spp", BOX, 64, 64, 4, 8),
        # A small scene at a useful sample count: many bounces in few triangles.
        _render("box_256x256_64spp", BOX, 256, 256, 64, 8),
        # The benchmark's frame: 262,144 triangles, 1080p, 16 samples, depth 12.
        _render("terrain_1080p_16spp", 262144, 1920, 1080, 16, 12),
        # An interactive preview of odd size through a thin lens, with a contribution clamp.
        _render("terrain_853x479_3spp_lens", 262144, 853, 479, 3, 5, camera="orbit", aperture=0.02, clamp=8.0),
        # Larger scenes of the serving configuration, one request each: the walk leaves the near caches.
        _render("terrain1m_720p_8spp", 1 << 20, 1280, 720, 8, 8, camera="orbit"),
        _render("terrain4m_640x360_8spp", 1 << 22, 640, 360, 8, 4),
        # A contact sheet: uneven views of one scene in one call.
        {"name": "views_12", "kind": "views", "triangles": 262144, "count": 12, "depth": 12},
        # A viewer's frames from a cut on: one sample each, denoised with history and displayed.
        {"name": "realtime_1600x900", "kind": "realtime", "triangles": 262144, "width": 1600, "height": 900, "frames": 4, "depth": 8},
        # A denoiser behind another renderer: its own G-buffers, two frames with history.
        {"name": "svgf_1600x900", "kind": "svgf", "width": 1600, "height": 900, "frames": 2, "passes": 5},
        {"name": "svgf_427x241", "kind": "svgf", "width": 427, "height": 241, "frames": 3, "passes": 4},
        # A burst of mixed requests at a render server holding two scenes.
        {"name": "server_20", "kind": "server", "triangles": 262144, "requests": 20},
        # A lighting edit: new emitters and sky on a resident scene, then a one-sample preview.
        {"name": "relight_640x360", "kind": "relight", "triangles": 262144, "width": 640, "height": 360},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case of the listed ranges; sizes are log-uniform and mostly odd."""
    kind = rng.choice(["render", "render", "render", "render", "views", "realtime", "svgf", "server", "relight"])
    tris = 2 * _log_int(rng, 1 << 15, 1 << 19)
    w = _log_int(rng, 64, 1920)
    h = max(36, int(w * rng.uniform(0.5, 1.0)))
    if kind == "render":
        box = rng.random() < 0.25
        spp = min(_log_int(rng, 1, 64), max(1, 1920 * 1080 * 4 // (w * h)))
        return {"kind": "render", "triangles": BOX if box else tris, "width": w, "height": h, "spp": spp, "depth": rng.randint(2, 12),
                "camera": "scene" if box else rng.choice(["scene", "orbit"]), "aperture": rng.choice([0.0, 0.0, 0.01]),
                "clamp": rng.choice([0.0, 0.0, 5.0])}
    if kind == "views":
        return {"kind": "views", "triangles": tris, "count": rng.randint(2, 12), "depth": rng.choice([4, 8, 12])}
    if kind == "server":
        return {"kind": "server", "triangles": tris, "requests": rng.randint(4, 20)}
    w, h = max(w, 160), max(h, 90)
    if kind == "realtime":
        return {"kind": "realtime", "triangles": tris, "width": w, "height": h, "frames": rng.randint(2, 5), "depth": rng.choice([4, 8, 12])}
    if kind == "svgf":
        return {"kind": "svgf", "width": w, "height": h, "frames": rng.randint(1, 3), "passes": rng.randint(1, 5)}
    return {"kind": "relight", "triangles": tris, "width": w, "height": h}


# ---- inputs ---------------------------------------------------------------------------------------------


def _scene(triangles, seed):
    g = native.box_scene() if triangles == BOX else native.terrain_scene(triangles, 1 + seed % 100003)
    return g, g.build(gpu=True)


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


def _resident(case, seed):
    g, b = _scene(case["triangles"], seed)
    r = native.Renderer(0)
    r.upload(b.desc)
    if "width" in case:
        r.resize(case["width"], case["height"])
    return g, b, r


def _view_sizes(case):
    """Width, height and spp of each view of a set, or of each request of a burst, mixed."""
    rng = random.Random(7)
    out = []
    if case["kind"] == "views":
        n = case["count"]
        for k in range(n):
            w = int(round(320 * 6 ** ((k + rng.random()) / n)))
            out.append((w, max(180, int(round(w * 9 / 16))), (1, 4, 16, 4)[k % 4]))
    else:
        for k in range(case["requests"]):
            w, h = workloads.RESOLUTIONS[(0, 0, 1, 0, 1, 2, 0, 1, 3, 2)[k % 10]]
            out.append((w, h, (1, 8, 4)[k % 3]))
    rng.shuffle(out)
    return out


def _relight(g, seed):
    """New emission, punctual intensities and sky for the generated scene `g` (abi.LightUpdate and what it points to)."""
    raw, rng = g.raw, np.random.default_rng(seed)
    mats = (abi.Material * raw.num_materials)()
    C.memmove(mats, raw.materials, C.sizeof(abi.Material) * raw.num_materials)
    for m in mats:
        f = float(rng.uniform(0.2, 5.0))
        m.emission = abi.Vec3(m.emission.x * f, m.emission.y * f, m.emission.z * f)
    punct = (abi.PunctualLight * max(1, raw.num_punctual))()
    if raw.num_punctual:
        C.memmove(punct, raw.punctual, C.sizeof(abi.PunctualLight) * raw.num_punctual)
    n = raw.env_width * raw.env_height
    env = np.ctypeslib.as_array(C.cast(raw.env_texels, C.POINTER(C.c_float)), shape=(n * 3,)).copy()
    env = np.roll(env.reshape(raw.env_height, raw.env_width, 3), int(rng.integers(raw.env_width)), axis=1)
    env = np.ascontiguousarray(env * rng.uniform(0.3, 2.0, (1, 1, 3)).astype(np.float32), np.float32)
    u = abi.LightUpdate(C.cast(mats, C.POINTER(abi.Material)), raw.num_materials, C.cast(punct, C.POINTER(abi.PunctualLight)),
                        raw.num_punctual, env.ctypes.data_as(C.POINTER(abi.Vec3)), raw.env_width, raw.env_height, raw.env_color,
                        raw.env_intensity, raw.env_rotation + float(rng.uniform(0, 1)))
    return u, (mats, punct, env)


def _svgf_cameras(case, seed):
    a = 0.02 * (seed % 300)
    w, h = case["width"], case["height"]
    return [workloads.look_at((6 * math.cos(a + 0.01 * k), 2.5, 6 * math.sin(a + 0.01 * k)), (0, 0.8, 0), 45.0, w / h)
            for k in range(case["frames"])]


def _svgf_frames(case, seed, cams):
    """One-sample G-buffers (float4 images) of a floor and seven spheres under a sky, by analytic ray casts."""
    w, h = case["width"], case["height"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = random.Random(seed)
    spheres = [(rng.uniform(-3, 3), rng.uniform(0.3, 1.2), rng.uniform(-3, 3), rng.uniform(0.3, 0.9)) for _ in range(7)]
    f64 = dict(dtype=torch.float64, device="cuda")
    vec = lambda v: torch.tensor([v.x, v.y, v.z], **f64)  # noqa: E731
    tint = torch.rand((9, 3), generator=gen, **f64) * 0.8 + 0.1
    out = []
    for cam in cams:
        y, x = torch.meshgrid(torch.arange(h, **f64), torch.arange(w, **f64), indexing="ij")
        sx = (2 * (x + 0.5) / w - 1) * cam.tan_half_fov * cam.aspect
        sy = (1 - 2 * (y + 0.5) / h) * cam.tan_half_fov
        d = vec(cam.forward) + sx[..., None] * vec(cam.right) + sy[..., None] * vec(cam.up)
        d = d / d.norm(dim=-1, keepdim=True)
        o = vec(cam.position)
        t = torch.where(d[..., 1] < -1e-6, -o[1] / d[..., 1], torch.inf)
        t = torch.where(t < 40, t, torch.inf)
        mat = torch.where(torch.isfinite(t), 0, -1)
        n = torch.zeros_like(d)
        n[..., 1] = 1
        for k, (cx, cy, cz, r) in enumerate(spheres):
            oc = o - torch.tensor([cx, cy, cz], **f64)
            b = (d * oc).sum(-1)
            q = b * b - (oc @ oc - r * r)
            ts = -b - q.clamp_min(0).sqrt()
            hit = (q > 0) & (ts > 1e-3) & (ts < t)
            t = torch.where(hit, ts, t)
            mat = torch.where(hit, k + 1, mat)
            n = torch.where(hit[..., None], (oc + ts[..., None] * d) / r, n)
        miss = mat < 0
        t = torch.where(miss, 0.0, t)
        p = o + torch.where(miss, 1e4, t)[..., None] * d
        checker = 0.6 + 0.4 * ((p[..., 0].floor() + p[..., 2].floor()) % 2)
        albedo = torch.where(miss[..., None], 1.0, tint[mat.clamp_min(0)] * checker[..., None])
        glow = torch.where((mat == 3)[..., None], 2.0 * tint[3], 0.0)
        sky = 0.4 + 0.6 * d[..., 1:2].abs() * torch.tensor([0.6, 0.8, 1.0], **f64)
        emission = torch.where(miss[..., None], sky, glow)
        light = (n[..., 1:2] * 0.5 + 0.6) * torch.empty((h, w, 1), **f64).exponential_(1.0, generator=gen)
        color = torch.where(miss[..., None], sky, albedo * light + emission)
        four = lambda a, last: torch.cat([a, last.expand(h, w, 1) if last.dim() < 3 else last], -1).float().contiguous()  # noqa: E731
        one = torch.ones((h, w, 1), **f64)
        out.append({"color": four(color, one), "albedo": four(albedo, one),
                    "normal_depth": four(torch.where(miss[..., None], -d, n), t[..., None]),
                    "position": four(p, mat[..., None].double()), "emission": four(emission, one)})
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "svgf":
        s["cams"] = _svgf_cameras(case, seed)
        s["frames"] = _svgf_frames(case, seed, s["cams"])
        s["out"] = [torch.zeros((case["height"], case["width"], 4), device="cuda") for _ in s["frames"]]
        s["svgf"] = native.Svgf(case["width"], case["height"])
        s["settings"] = abi.svgf_settings(atrous_iterations=case["passes"])
        return s
    if kind == "server":
        box, terrain = _scene(BOX, seed), _scene(case["triangles"], seed)
        s["server"] = native.Server(budget_bytes=32 << 30)
        s["scenes"] = [s["server"].add_scene(b.desc) for _, b in (box, terrain)]
        rng = np.random.default_rng(seed)
        center, extent = workloads.scene_sphere(terrain[1].desc)
        s["requests"] = []
        for k, (w, h, spp) in enumerate(_view_sizes(case)):
            cam = box[0].camera(w / h) if k % 4 == 0 else workloads.sphere_camera(rng, center, 0.5 * extent, w / h)
            s["requests"].append((s["scenes"][0 if k % 4 == 0 else 1], cam, w, h, spp, seed + k, abi.path_options(max_depth=(4, 8, 12)[k % 3])))
        return s
    g, b, r = _resident(case, seed)
    s.update(renderer=r, keep=(g, b))
    if kind == "views":
        rng = np.random.default_rng(seed)
        center, extent = workloads.scene_sphere(b.desc)
        s["views"] = [abi.View(workloads.sphere_camera(rng, center, 0.6 * extent, w / h), w, h, spp, seed + k,
                               abi.path_options(max_depth=case["depth"]))
                      for k, (w, h, spp) in enumerate(_view_sizes(case))]
        return s
    w, h = case["width"], case["height"]
    s["rs"] = abi.render_settings(w, h, max_depth=case.get("depth", 8), clamp=case.get("clamp", 0.0), seed=seed & 0x7fffffff)
    if kind == "realtime":
        s["cams"] = workloads.orbit_cameras(b.desc, case["frames"], w / h, start_deg=seed % 360)
        s["settings"] = abi.svgf_settings()
    else:
        if case.get("camera") == "orbit":
            s["cam"] = workloads.orbit_cameras(b.desc, 1, w / h, start_deg=seed % 360, radius=0.4, elevation=0.15)[0]
        else:
            s["cam"] = g.camera(w / h)
        s["cam"].aperture = case.get("aperture", 0.0)
        s["image"] = _pinned(h, w, 3)
        if kind == "relight":
            s["update"], s["lights"] = _relight(g, seed)
    return s


# ---- one pass -------------------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "svgf":
        sv, cams = state["svgf"], state["cams"]
        sv.reset()
        for k, (f, out) in enumerate(zip(state["frames"], state["out"])):
            sv.run(f["color"].data_ptr(), f["albedo"].data_ptr(), f["normal_depth"].data_ptr(), f["position"].data_ptr(),
                   f["emission"].data_ptr(), cams[max(k - 1, 0)], state["settings"], out.data_ptr())
        return state["out"]
    if kind == "server":
        srv = state["server"]
        ids = [srv.submit(sid, cam, w, h, spp, seed, path) for sid, cam, w, h, spp, seed, path in state["requests"]]
        images = []
        for rid, q in zip(ids, state["requests"]):
            srv.wait(rid)
            images.append(srv.fetch(rid, q[2], q[3])[0])
        return images
    r = state["renderer"]
    if kind == "views":
        r.render_views(state["views"])
        return [r.download_view(k, v.width, v.height) for k, v in enumerate(state["views"])]
    if kind == "realtime":
        r.reset()
        cams = state["cams"]
        for k, cam in enumerate(cams):
            r.render_denoised(cam, cams[max(k - 1, 0)], state["rs"], state["settings"])
            r.display(state["rs"])
        return {"image": r.download_image(), "display": r.download_display()}
    if kind == "relight":
        r.rebuild_lights(state["update"])
    r.reset()
    r.render(state["cam"], state["rs"], case.get("spp", 1))
    return r.download_image(out=state["image"])


# ---- what a pass cannot do without ----------------------------------------------------------------------

_RAYS = {True: 9.0, False: 2.2}  # closest-hit and shadow rays a sample takes: in the closed box, in the open scenes


def _trace_work(triangles, samples, pixels):
    """A ray meets the two child boxes (some 20 operations each) of about two nodes per level of the tree and about ten
    triangles (some 45 each); the scene's nodes and triangles (64 and 48 bytes, half as many nodes) are read and the
    image written."""
    visits = 2 * math.log2(triangles)
    rays = samples * _RAYS[triangles == BOX]
    return {"bytes": triangles * 80.0 + 12.0 * pixels, "flops": rays * (visits * 2 * 20 + 10 * 45)}


def work(case):
    kind = case["kind"]
    if kind == "svgf" or kind == "realtime":
        px = case["width"] * case["height"] * case["frames"]
        passes = case.get("passes", 5)
        # Five input images and the output; a frame's filter taps: 49 of some 30 operations and 25 of some 50 per pass.
        sv = {"bytes": px * 16.0 * 6, "flops": px * (25.0 * 50 * passes + 49 * 30)}
        if kind == "svgf":
            return sv
        tr = _trace_work(case["triangles"], px, px)
        return {k: sv[k] + tr[k] for k in sv}
    if kind in ("views", "server"):
        sizes = _view_sizes(case)
        return _trace_work(case["triangles"], sum(w * h * n for w, h, n in sizes), sum(w * h for w, h, _ in sizes))
    px = case["width"] * case["height"]
    return _trace_work(case["triangles"], px * case.get("spp", 1), px)


# ---- the denoiser in 64 bits ----------------------------------------------------------------------------


def _shift(a, dx, dy, fill=0.0):
    """a[y + dy, x + dx], `fill` outside the image."""
    h, w = a.shape[:2]
    out = torch.full_like(a, fill)
    if abs(dx) < w and abs(dy) < h:
        out[max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)] = a[max(0, dy):h - max(0, -dy), max(0, dx):w - max(0, -dx)]
    return out


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _clamped(a, dx, dy):
    h, w = a.shape[:2]
    y = (torch.arange(h, device=a.device) + dy).clamp(0, h - 1)
    x = (torch.arange(w, device=a.device) + dx).clamp(0, w - 1)
    return a[y][:, x]


def _exact_svgf(frames, cams, passes, alpha=0.2, phi_color=4.0, phi_normal=128.0, phi_depth=1.0):
    outs, hist = [], None
    for k, f in enumerate(frames):
        color, albedo, nd, pos, em = (f[n].double() for n in ("color", "albedo", "normal_depth", "position", "emission"))
        h, w = color.shape[:2]
        n, z, mat = nd[..., :3] / nd[..., :3].norm(dim=-1, keepdim=True), nd[..., 3], pos[..., 3]
        surface = mat >= 0
        cur = (color - em)[..., :3].clamp_min(0) / albedo[..., :3].clamp_min(1e-3)
        lum = _lum(cur)
        c, m0, m1, length = cur, lum, lum * lum, torch.ones_like(lum)
        if hist is not None:
            pc = cams[k - 1]
            vec = lambda v: torch.tensor([v.x, v.y, v.z], dtype=torch.float64, device=z.device)  # noqa: E731
            d = pos[..., :3] - vec(pc.position)
            zz = d @ vec(pc.forward)
            ok = surface & (zz > 1e-4)
            zs = torch.where(ok, zz, 1.0)
            px = ((d @ vec(pc.right)) / (zs * pc.tan_half_fov * pc.aspect) + 1) * 0.5 * w - 0.5
            py = (1 - (d @ vec(pc.up)) / (zs * pc.tan_half_fov)) * 0.5 * h - 0.5
            dist = d.norm(dim=-1)
            x0, y0 = px.floor(), py.floor()
            fx, fy = px - x0, py - y0
            acc = torch.zeros((h, w, 6), dtype=torch.float64, device=z.device)
            wsum = torch.zeros_like(z)
            for q in range(4):
                xx, yy = x0 + (q & 1), y0 + (q >> 1)
                inside = ok & (xx >= 0) & (yy >= 0) & (xx < w) & (yy < h)
                j = (yy.clamp(0, h - 1) * w + xx.clamp(0, w - 1)).long()
                pn, pz, pm = hist["n"].reshape(-1, 3)[j], hist["z"].reshape(-1)[j], hist["mat"].reshape(-1)[j]
                keep = inside & (pm == mat) & ((pz - dist).abs() <= 0.05 * dist + 0.01) & ((pn * n).sum(-1) >= 0.9)
                bw = torch.where(keep, (fx if q & 1 else 1 - fx) * (fy if q >> 1 else 1 - fy), 0.0)
                acc += hist["v"].reshape(-1, 6)[j] * bw[..., None]
                wsum += bw
            use = wsum > 1e-3
            acc = acc / torch.where(use, wsum, 1.0)[..., None]
            len1 = (acc[..., 5] + 1).clamp_max(64)
            a = (1 / len1).clamp_min(alpha)
            mix = lambda old, new: old + (new - old) * a  # noqa: E731
            c = torch.where(use[..., None], acc[..., :3] + (cur - acc[..., :3]) * a[..., None], c)
            m0, m1 = torch.where(use, mix(acc[..., 3], lum), m0), torch.where(use, mix(acc[..., 4], lum * lum), m1)
            length = torch.where(use, len1, length)
        var = (m1 - m0 * m0).clamp_min(0)
        # The spatial estimate while the history is short.
        v7 = torch.cat([c, m0[..., None], m1[..., None]], -1)
        acc, wsum = torch.zeros_like(v7), torch.zeros_like(z)
        for dy in range(-3, 4):
            for dx in range(-3, 4):
                same = _shift(mat, dx, dy, -2.0) == mat
                cos = (_shift(n, dx, dy) * n).sum(-1).clamp_min(0)
                wt = torch.where(same, cos ** phi_normal * torch.exp(-(_shift(z, dx, dy) - z).abs() / (0.05 * z + 1e-3)), 0.0)
                acc += _shift(v7, dx, dy) * wt[..., None]
                wsum += wt
        short = surface & (length < 4) & (wsum > 0)
        acc = acc / torch.where(short, wsum, 1.0)[..., None]
        var = torch.where(short, (acc[..., 4] - acc[..., 3] ** 2).clamp_min(0) * (4 / length), var)
        src = torch.cat([torch.where(short[..., None], acc[..., :3], c), var[..., None]], -1)
        zx = _clamped(z, 1, 0) - _clamped(z, -1, 0)
        zy = _clamped(z, 0, 1) - _clamped(z, 0, -1)
        grad = 0.5 * torch.maximum(zx.abs(), zy.abs())
        for it in range(passes):
            step = 1 << it
            blur = sum(_clamped(src[..., 3], dx, dy) * (0.25 if dx == dy == 0 else 0.125 if dx * dy == 0 else 0.0625)
                       for dx in (-1, 0, 1) for dy in (-1, 0, 1))
            sigma = phi_color * blur.clamp_min(0).sqrt() + 1e-4
            lc = _lum(src)
            acc, vsum, wsum = torch.zeros_like(src[..., :3]), torch.zeros_like(z), torch.zeros_like(z)
            for dy in range(-2, 3):
                for dx in range(-2, 3):
                    sx, sy = dx * step, dy * step
                    same = _shift(mat, sx, sy, -2.0) == mat
                    s = _shift(src, sx, sy)
                    kern = (3 / 8, 1 / 4, 1 / 16)[abs(dx)] * (3 / 8, 1 / 4, 1 / 16)[abs(dy)]
                    cos = (_shift(n, sx, sy) * n).sum(-1).clamp_min(0)
                    den = phi_depth * grad * step * math.hypot(dx, dy) + 1e-3 * z + 1e-4
                    wt = kern * cos ** phi_normal * torch.exp(-(_lum(s) - lc).abs() / sigma - (_shift(z, sx, sy) - z).abs() / den)
                    wt = torch.where(same, wt, 0.0)
                    acc += s[..., :3] * wt[..., None]
                    vsum += wt * wt * s[..., 3]
                    wsum += wt
            done = surface & (wsum > 0)
            ws = torch.where(done, wsum, 1.0)
            src = torch.where(done[..., None], torch.cat([acc / ws[..., None], (vsum / (ws * ws))[..., None]], -1), src)
            if it == 0:
                hist = {"n": n, "z": z, "mat": mat,
                        "v": torch.cat([src[..., :3], m0[..., None], m1[..., None], length[..., None]], -1)}
        out = src[..., :3] * albedo[..., :3].clamp_min(1e-3) + em[..., :3]
        out = torch.cat([out, torch.ones_like(out[..., :1])], -1)
        outs.append(torch.where(surface[..., None], out, color))
    return outs


def exact(case, seed):
    if case["kind"] != "svgf":
        return None
    cams = _svgf_cameras(case, seed)
    return _exact_svgf(_svgf_frames(case, seed, cams), cams, case["passes"])
