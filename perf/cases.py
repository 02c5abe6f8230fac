"""The work users of dort_b200 have it do, as cases that can be timed.

A case is a dict of plain values.  ``listed()`` names the usual ones,
``draw(rng)`` makes another one of the same ranges, ``prepare`` builds what a
program holds before the call (device scene, rays or render parameters, output
buffers), ``run`` is one pass through the public entry points, ``work`` its
unavoidable bytes and operations, ``exact`` the ray casts' results in 64 bits.

Kinds of work:

* ``cast``    Scene.raycast_device: closest or any hit of rays in device
              memory (picking, visibility and occlusion queries, baking);
* ``rebuild`` Scene(...) on changed geometry, then a cast (animation);
* ``frame``   the path tracer's wavefront on one image;
* ``render``  Scene.render_device with the path, light or bidirectional
              tracer;
* ``batch``   many scenes in one wavefront launch;
* ``adjoint`` one step of an inverse-rendering loop: forward image, loss,
              gradients.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dort_b200 as db
from dort_b200 import scenes

# float32 values of a ray: origin, t_min, direction, t_max
RAY = 8
MISS = -1          # 0xffffffff as int32


def listed():
    return [
        # a viewport's pick / line-of-sight query: the launch is what it costs
        {"name": "cast_pick", "kind": "cast", "geometry": "soup", "tris": 20_000, "rays": 4_096,
         "rays_of": "mixed", "any_hit": False, "watertight": False},
        # the benchmark's ray cast: 1M-triangle soup, half camera rays, half
        # diffuse bounces
        {"name": "cast_16m", "kind": "cast", "geometry": "soup", "tris": 1_000_000,
         "rays": 16_777_216, "rays_of": "mixed", "any_hit": False, "watertight": False},
        # occlusion baking over a mesh: any hit towards a light, a ragged count
        {"name": "cast_shadow", "kind": "cast", "geometry": "sphere", "tris": 250_882,
         "rays": 3_000_001, "rays_of": "shadow", "any_hit": True, "watertight": False},
        # a closed mesh queried with the watertight test, ragged count
        {"name": "cast_watertight", "kind": "cast", "geometry": "sphere", "tris": 92_482,
         "rays": 700_001, "rays_of": "bounce", "any_hit": False, "watertight": True},
        # geometry that changed since the last frame: build, then query
        {"name": "rebuild_500k", "kind": "rebuild", "geometry": "soup", "tris": 500_000,
         "rays": 262_144, "rays_of": "mixed", "any_hit": False, "watertight": False},
        # a preview while a scene is edited: small odd image, one sample
        {"name": "frame_preview", "kind": "frame", "scene": "cornell_delt", "freq": 0,
         "width": 161, "height": 91, "spp": 1, "depth": 5},
        # the Cornell box of the reference's tests
        {"name": "frame_cornell", "kind": "frame", "scene": "cornell_diff", "freq": 0,
         "width": 256, "height": 256, "spp": 64, "depth": 8},
        # the benchmark's 1080p frame (2M-triangle displaced sphere under a
        # sky), at the samples of one progressive pass
        {"name": "frame_1080p", "kind": "frame", "scene": "sphere_sky", "freq": 316,
         "width": 1920, "height": 1080, "spp": 16, "depth": 16},
        # everything the general code path has: shapes, point light, thin
        # lens, glossy and rough materials, one kernel for the whole path
        {"name": "render_general", "kind": "render", "renderer": "pt", "scene": "general",
         "freq": 0, "width": 200, "height": 150, "spp": 32, "depth": 6},
        # the light and the bidirectional tracer on the Cornell box are the
        # reference's other integrators
        {"name": "render_bdpt", "kind": "render", "renderer": "bdpt", "scene": "cornell_glos",
         "freq": 0, "width": 256, "height": 256, "spp": 16, "depth": 8},
        # a data-set job: many small scenes of different sizes at once
        {"name": "batch_16", "kind": "batch", "jobs": 16, "min_tris": 10_000, "max_tris": 100_000,
         "min_res": 48, "max_res": 256, "spp": 24, "depth": 10},
        # inverse rendering: per-triangle albedo and emission gradients
        {"name": "adjoint_step", "kind": "adjoint", "tris": 200_000, "width": 256, "height": 256,
         "spp": 32, "depth": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "cast", "rebuild", "frame", "frame", "frame", "render",
                       "render", "batch", "adjoint"])
    if kind in ("cast", "rebuild"):
        geometry = rng.choice(["soup", "sphere"])
        rays_of = rng.choice(["camera", "bounce", "mixed", "shadow"])
        if kind == "cast":
            tris, rays = _log_int(rng, 1_000, 1_000_000), _log_int(rng, 1_000, 16_000_000)
        else:
            tris, rays = _log_int(rng, 5_000, 500_000), _log_int(rng, 1_000, 250_000)
        if geometry == "sphere":
            freq = max(5, int(math.sqrt(tris / 20)))
            tris = 20 * freq * freq + 2
        return {"kind": kind, "geometry": geometry, "tris": tris, "rays": rays,
                "rays_of": rays_of, "any_hit": rays_of == "shadow" or rng.random() < 0.15,
                "watertight": rng.random() < 0.25}
    if kind == "frame":
        scene = rng.choice(["cornell_diff", "cornell_glos", "cornell_delt", "sphere_sky",
                            "sphere_sky"])
        freq = _log_int(rng, 12, 200) if scene == "sphere_sky" else 0
        w, h = _log_int(rng, 48, 1_600), _log_int(rng, 40, 1_000)
        spp = max(1, min(256, _log_int(rng, 40_000, 20_000_000) // (w * h)))
        return {"kind": "frame", "scene": scene, "freq": freq, "width": w, "height": h,
                "spp": spp, "depth": rng.randint(2, 16)}
    if kind == "render":
        renderer = rng.choice(["pt", "lt", "bdpt"])
        scene = rng.choice(["cornell_diff", "cornell_glos", "general"])
        w, h = _log_int(rng, 40, 400), _log_int(rng, 40, 400)
        spp = max(1, min(128, _log_int(rng, 20_000, 2_000_000) // (w * h)))
        return {"kind": "render", "renderer": renderer, "scene": scene, "freq": 0, "width": w,
                "height": h, "spp": spp, "depth": rng.randint(2, 8)}
    if kind == "batch":
        lo = _log_int(rng, 40, 100)
        return {"kind": "batch", "jobs": rng.randint(2, 24), "min_tris": 2_000,
                "max_tris": _log_int(rng, 10_000, 100_000), "min_res": lo,
                "max_res": lo + rng.randint(10, 150), "spp": rng.randint(1, 32),
                "depth": rng.randint(4, 16)}
    w, h = _log_int(rng, 48, 256), _log_int(rng, 48, 256)
    return {"kind": "adjoint", "tris": _log_int(rng, 2_000, 200_000), "width": w, "height": h,
            "spp": rng.randint(2, 32), "depth": rng.randint(2, 6)}


# ---- inputs ----------------------------------------------------------------------

def _geometry(case, seed):
    """Host arrays (verts, tris) and the eye and target of a camera on them."""
    if case["geometry"] == "soup":
        # the benchmark's soup holds 1M triangles of edge sigma 0.01: the same
        # density of surface for other counts
        sigma = 0.01 * math.sqrt(1_000_000 / max(case["tris"], 10_000))
        verts, tris = scenes.random_triangles(case["tris"], seed=seed, sigma=min(sigma, 0.1))
        return verts, tris, (0.5, 0.5, -1.6), (0.5, 0.5, 0.5)
    freq = int(round(math.sqrt((case["tris"] - 2) / 20)))
    d = scenes.wavefront_scene(freq, sky_w=8, sky_h=4, seed=seed)
    return d["verts"], d["tris"], (0.0, 1.6, -4.2), (0.0, 1.05, 0.0)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _camera_rays(n, eye, target):
    """n rays through the pixel centres of a 2:1 image, row-major."""
    dev = "cuda"
    h = max(1, int(math.sqrt(n / 2)))
    w = -(-n // h)
    i = torch.arange(n, device=dev)
    x = ((i % w).double() + 0.5) / w * 2 - 1
    y = 1 - ((i // w).double() + 0.5) / h * 2
    eye_t = torch.tensor(eye, dtype=torch.float64, device=dev)
    fwd = _unit(torch.tensor(target, dtype=torch.float64, device=dev) - eye_t)
    right = _unit(torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64,
                                                       device=dev)))
    up = torch.linalg.cross(right, fwd)
    tan_h = math.tan(math.radians(40.0) / 2)
    d = _unit(fwd + (x * tan_h)[:, None] * right + (y * tan_h / 2)[:, None] * up)
    rays = torch.empty(n, RAY, dtype=torch.float32, device=dev)
    rays[:, 0:3] = eye_t.float()
    rays[:, 3] = 0.0
    rays[:, 4:7] = d.float()
    rays[:, 7] = math.inf
    return rays


def _surface_points(n, verts, tris, eye, target, gen):
    """n points on the geometry in image order (as the hits of a picture's
    pixels come, row of tiles by row of tiles), and the unit normals facing
    the eye."""
    dev = "cuda"
    v = torch.from_numpy(verts).to(dev)
    t = torch.from_numpy(tris.astype(np.int64)).to(dev)
    # the last two triangles of the sphere scene are its 40 x 40 ground
    pick = torch.randint(0, max(1, len(tris) - 2), (n,), generator=gen, device=dev)
    b = torch.rand(n, 2, generator=gen, device=dev)
    b = torch.where((b.sum(1) > 1)[:, None], 1 - b, b)
    p0, p1, p2 = v[t[pick, 0]], v[t[pick, 1]], v[t[pick, 2]]
    p = p0 + b[:, :1] * (p1 - p0) + b[:, 1:] * (p2 - p0)
    nn = torch.linalg.cross(p2 - p0, p1 - p0)
    nn = nn / nn.norm(dim=1, keepdim=True).clamp_min(1e-20)
    eye_t = torch.tensor(eye, dtype=torch.float32, device=dev)
    fwd = _unit(torch.tensor(target, dtype=torch.float32, device=dev) - eye_t)
    right = _unit(torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device=dev)))
    up = torch.linalg.cross(right, fwd)
    to = p - eye_t
    nn = torch.where(((nn * to).sum(1) > 0)[:, None], -nn, nn)
    z = (to @ fwd).clamp_min(1e-3)
    px = ((to @ right) / z * 600).long().clamp(-4095, 4095) + 4096
    py = (-(to @ up) / z * 600).long().clamp(-4095, 4095) + 4096
    order = torch.argsort(((py // 4) * 8192 + px // 8) * 32 + (py % 4) * 8 + px % 8, stable=True)
    return p[order], nn[order], to.norm(dim=1)[order]


def _bounce_rays(n, verts, tris, eye, target, gen):
    """Cosine-distributed rays leaving the surface points, t_min a thousandth
    of the distance to the eye (the reference's ray epsilon)."""
    p, nn, dist = _surface_points(n, verts, tris, eye, target, gen)
    u = torch.rand(n, 2, generator=gen, device="cuda")
    r, phi = u[:, 0].sqrt(), 2 * math.pi * u[:, 1]
    a = torch.where((nn[:, 0].abs() > 0.7)[:, None], torch.tensor([0.0, 1.0, 0.0], device="cuda"),
                    torch.tensor([1.0, 0.0, 0.0], device="cuda"))
    tx = _unit(torch.linalg.cross(a, nn))
    ty = torch.linalg.cross(nn, tx)
    d = ((r * phi.cos())[:, None] * tx + (r * phi.sin())[:, None] * ty +
         (1 - u[:, 0]).clamp_min(0).sqrt()[:, None] * nn)
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-20)
    rays = torch.empty(n, RAY, dtype=torch.float32, device="cuda")
    rays[:, 0:3] = p
    rays[:, 3] = 1e-3 * dist
    rays[:, 4:7] = d
    rays[:, 7] = math.inf
    return rays


def _shadow_rays(n, verts, tris, eye, target, gen):
    """Segments from the surface points to points on a square light above."""
    p, _, dist = _surface_points(n, verts, tris, eye, target, gen)
    u = torch.rand(n, 2, generator=gen, device="cuda")
    top = float(verts[: max(1, len(verts) - 4), 1].max()) + 1.0
    q = torch.stack([target[0] + u[:, 0] - 0.2, torch.full((n,), top, device="cuda"),
                     target[2] + u[:, 1] - 0.8], 1)
    d = q - p
    far = d.norm(dim=1)
    rays = torch.empty(n, RAY, dtype=torch.float32, device="cuda")
    rays[:, 0:3] = p
    rays[:, 3] = 1e-3 * dist
    rays[:, 4:7] = d / far[:, None]
    rays[:, 7] = far * 0.999
    return rays


def _rays(case, seed, verts, tris, eye, target):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, of = case["rays"], case["rays_of"]
    if of == "camera":
        return _camera_rays(n, eye, target)
    if of == "bounce":
        return _bounce_rays(n, verts, tris, eye, target, gen)
    if of == "shadow":
        return _shadow_rays(n, verts, tris, eye, target, gen)
    half = n // 2
    return torch.cat([_camera_rays(half, eye, target),
                      _bounce_rays(n - half, verts, tris, eye, target, gen)]).contiguous()


def _general_scene(seed):
    """A Cornell box with glossy boxes, a glass and a rough sphere, a disk, a
    point light beside the area light, and a thin-lens camera."""
    rng = np.random.default_rng(seed)
    c = scenes.cornell_variant("glos", "both")
    mats = c["materials"]
    glass, rough, metal = len(mats), len(mats) + 1, len(mats) + 2
    mats += [{"kind": db.MAT_DIELECTRIC, "color": (1.0, 1.0, 1.0), "color2": (1.0, 1.0, 1.0),
              "param": (1.5,)},
             {"kind": db.MAT_OREN_NAYAR, "color": (0.4, 0.5, 0.6), "param": (0.3,)},
             {"kind": db.MAT_CONDUCTOR, "color": (0.9, 0.7, 0.4), "param": (0.2,)}]

    def at(x, y, z):
        return [[1.0, 0.0, 0.0, x], [0.0, 1.0, 0.0, y], [0.0, 0.0, 1.0, z]]

    jitter = rng.uniform(-0.2, 0.2, 4)
    c["shapes"] = [
        {"kind": db.SHAPE_SPHERE, "material": glass, "param": (0.5,),
         "to_world": at(4.2 + jitter[0], 0.6, 1.0)},
        {"kind": db.SHAPE_SPHERE, "material": rough, "param": (0.4,),
         "to_world": at(1.0 + jitter[1], 0.5, 3.6)},
        {"kind": db.SHAPE_SPHERE, "material": metal, "param": (0.45,),
         "to_world": at(1.85, 2.1 + jitter[2], 1.7)},
    ]
    c["delta_lights"] = [{"kind": db.LIGHT_POINT, "rgb": (6.0, 6.0, 7.0),
                          "vec": (1.0 + jitter[3], 4.5, 1.0)}]
    c["camera"] = dict(c["camera"], kind=db.CAMERA_THIN_LENS, lens_radius=0.05,
                       focal_distance=10.0)
    return c


def _scene_dict(case, seed):
    name = case["scene"]
    if name == "sphere_sky":
        return scenes.wavefront_scene(case["freq"], seed=seed)
    if name == "general":
        return _general_scene(seed)
    return scenes.cornell_variant(name.split("_")[1])


def _adjoint_case(case, seed):
    d = scenes.adjoint_scene(case["tris"], seed=seed)
    rng = np.random.default_rng(seed + 1)
    target = rng.uniform(0.0, 0.5, (case["height"], case["width"], 3)).astype(np.float32)
    return d, target


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("cast", "rebuild"):
        verts, tris, eye, target = _geometry(case, seed)
        rays = _rays(case, seed, verts, tris, eye, target)
        st = {"case": case, "rays": rays,
              "prim": torch.zeros(case["rays"], dtype=torch.int32, device="cuda"),
              "tb": None if case["any_hit"]
              else torch.zeros(case["rays"], 3, dtype=torch.float32, device="cuda")}
        if kind == "cast":
            st["scene"] = db.Scene(verts, tris, watertight=case["watertight"])
        else:
            st["verts"], st["tris"] = verts, tris
        return st
    if kind in ("frame", "render"):
        d = _scene_dict(case, seed)
        params = db.render_params(d["camera"], case["width"], case["height"], case["spp"],
                                  max_depth=case["depth"], seed=seed,
                                  renderer=case.get("renderer", "pt"))
        return {"case": case, "scene": db.scene_from_dict(d), "params": params,
                "out": torch.zeros(case["height"], case["width"], 3, device="cuda")}
    if kind == "batch":
        # the sizes are the case's, the geometry the seed's
        rng = np.random.default_rng(case["jobs"] * 1000 + case["max_res"])
        held = []
        for k in range(case["jobs"]):
            n, w, h = (int(np.exp(rng.uniform(np.log(lo), np.log(hi))))
                       for lo, hi in ((case["min_tris"], case["max_tris"]),
                                      (case["min_res"], case["max_res"]),
                                      (case["min_res"], case["max_res"])))
            d = scenes.soup_with_light(n, seed + k)
            held.append((db.scene_from_dict(d),
                         db.render_params(d["camera"], w, h, case["spp"],
                                          max_depth=case["depth"], seed=seed + k)))
        return {"case": case, "batch": db.Batch(held), "held": held}
    d, target = _adjoint_case(case, seed)
    params = db.render_params(d["camera"], case["width"], case["height"], case["spp"],
                              max_depth=case["depth"], seed=seed)
    return {"case": case, "scene": db.scene_from_dict(d), "params": params, "target": target,
            "albedo": d["tri_albedo"], "emission": d["tri_emission"]}


# ---- one pass --------------------------------------------------------------------

def _cast(scene, st, case):
    scene.raycast_device(st["rays"].data_ptr(), case["rays"], st["prim"].data_ptr(),
                         None if st["tb"] is None else st["tb"].data_ptr(),
                         any_hit=case["any_hit"], stream=torch.cuda.current_stream().cuda_stream)
    return [st["prim"]] if st["tb"] is None else [st["prim"], st["tb"]]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "cast":
        return _cast(state["scene"], state, case)
    if kind == "rebuild":
        scene = db.Scene(state["verts"], state["tris"], watertight=case["watertight"])
        out = _cast(scene, state, case)
        scene.close()
        return out
    if kind == "frame":
        state["scene"].render_wavefront_device(state["params"], state["out"].data_ptr(),
                                               torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "render":
        state["scene"].render_device(state["params"], state["out"].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "batch":
        state["batch"].render(torch.cuda.current_stream().cuda_stream)
        return [state["batch"].image(j) for j in range(case["jobs"])]
    image = state["scene"].adjoint_forward(state["params"], tri_albedo=state["albedo"],
                                           tri_emission=state["emission"])
    loss, grad = db.loss_l2(image, state["target"])
    d_albedo, d_emission = state["scene"].adjoint_backward(state["params"], grad,
                                                           tri_albedo=state["albedo"],
                                                           tri_emission=state["emission"])
    return {"image": image, "loss": loss, "d_albedo": d_albedo, "d_emission": d_emission}


# ---- the work a pass cannot do without ---------------------------------------------

def _ray_flops(tris):
    """One descent of an 8-wide tree (12 operations a box) and one triangle
    test."""
    return 8 * 12 * math.ceil(math.log(max(tris, 8), 8)) + 50


def work(case):
    kind = case["kind"]
    if kind in ("cast", "rebuild"):
        out = 4 if case["any_hit"] else 16
        return {"bytes": case["rays"] * (4 * RAY + out) + 36 * case["tris"],
                "flops": case["rays"] * _ray_flops(case["tris"])}
    if kind == "batch":
        # the mean of the log-uniform sizes
        tris = math.sqrt(case["min_tris"] * case["max_tris"])
        res = math.sqrt(case["min_res"] * case["max_res"])
        samples = case["jobs"] * res * res * case["spp"]
        # a camera path meets two vertices at the least, each with a
        # continuation ray and a shadow ray
        return {"bytes": case["jobs"] * (36 * tris + 12 * res * res),
                "flops": samples * 4 * _ray_flops(tris)}
    pixels = case["width"] * case["height"]
    if kind == "adjoint":
        # forward and backward; image, target, albedo, both gradients
        return {"bytes": 36 * case["tris"] + 36 * pixels + 36 * case["tris"],
                "flops": 2 * pixels * case["spp"] * 4 * _ray_flops(case["tris"])}
    tris = 20 * case["freq"] ** 2 + 2 if case["scene"] == "sphere_sky" else 36
    return {"bytes": 48 * tris + 12 * pixels,
            "flops": pixels * case["spp"] * 4 * _ray_flops(tris)}


# ---- 64 bits ---------------------------------------------------------------------

def exact(case, seed):
    """t, b1, b2 of the ray casts by testing every triangle in 64 bits; None
    for the hit ids and for everything that is an estimate."""
    if case["kind"] not in ("cast", "rebuild") or case["any_hit"]:
        return None
    if case["rays"] * case["tris"] > 1e10:
        return None
    verts, tris, eye, target = _geometry(case, seed)
    rays = _rays(case, seed, verts, tris, eye, target).double()
    v = torch.from_numpy(verts).cuda().double()
    t = torch.from_numpy(tris.astype(np.int64)).cuda()
    p0 = v[t[:, 0]].T.contiguous()[:, None, :]
    e1 = (v[t[:, 1]] - v[t[:, 0]]).T.contiguous()[:, None, :]
    e2 = (v[t[:, 2]] - v[t[:, 0]]).T.contiguous()[:, None, :]

    def cross(a, b):
        return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    tb = torch.zeros(case["rays"], 3, dtype=torch.float64, device="cuda")
    step = max(1, int(1e8 // case["tris"]))
    for at in range(0, case["rays"], step):
        r = rays[at:at + step].T[:, :, None]
        o, lo, d, hi = r[0:3], r[3], r[4:7], r[7]
        s1 = cross(d, e2)
        inv = 1.0 / dot(s1, e1)
        s = o - p0
        b1 = dot(s1, s) * inv
        s2 = cross(s, e1)
        b2 = dot(s2, d) * inv
        th = dot(s2, e2) * inv
        ok = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (th >= lo) & (th <= hi)
        th = torch.where(ok, th, math.inf)
        best, k = th.min(dim=1)
        hit = torch.isfinite(best)
        found = torch.stack([best, b1.gather(1, k[:, None])[:, 0],
                             b2.gather(1, k[:, None])[:, 0]], 1)
        tb[at:at + step] = torch.where(hit[:, None], found, 0.0)
    return [None, tb]
