"""The work that a user has this framework do, as cases that can be timed.

Each case is one pass through the public entry points (``splat_gb300.tracer``,
``splat_gb300.batch``) under the library's default settings, at the sizes of
the repository's own workloads (``splat_gb300.scenes``), their tests and the
range in between:

* ``frame``    -- the fused forward step of one frame (``TraceStep.run``);
* ``animated`` -- a frame whose geometry moved: GPU rebuild of the BVH, then
  the step;
* ``render``   -- a whole ``trace!`` frame: forward step, camera pass, image;
* ``hits``     -- the nearest hit of a caller's rays in a resident scene;
* ``ntris``    -- the reference's brute-force hitter over its own triangle
  records;
* ``dropin``   -- the reference's ``trace!`` forward sequence on caller-owned
  ray records (``rays_from_light``, ``run_evolution``, ``continuum_light_map2``);
* ``steps``    -- the same frame with the reference's bounce loop kept on the
  caller's side: hit, evolve, partition, one call each per bounce;
* ``camera``   -- the reference's backward half on caller-owned records
  (``camera_rays``, ``run_evolution``, ``continuum_shade``);
* ``batch``    -- many uneven frames replayed as captured graphs.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from splat_gb300 import batch, scenes as S, tracer, types as T

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # a preview frame: 64 x 64 light grid on a 320-triangle lens; launches and latency count
        dict(name="frame_preview", kind="frame", scene="sphere", level=2, res1=64, res2=64, upscale=2, depth=3,
             planes=4, map_w=64, map_h=64, accum="i32", hitter="brute", material="cauchy"),
        # the smallest of the three named workloads: brute force, each ray at its own wavelength, float map
        dict(name="frame_plain", kind="frame", scene="sphere", level=5, res1=256, res2=256, upscale=1, depth=3,
             planes=0, map_w=256, map_h=256, accum="f32", hitter="brute", material="cauchy"),
        # the real-time workload: a displaced sphere, 2^20 rays splatted at 2 x 2 offsets into 16 planes
        dict(name="frame_realtime", kind="frame", scene="displaced", level=6, res1=2048, res2=2048, upscale=2,
             depth=4, planes=16, map_w=1024, map_h=1024, accum="i32", hitter="bvh", material="cauchy"),
        # the largest: 2^22 rays through a glass Menger sponge in a box, depth 6
        dict(name="frame_menger", kind="frame", scene="menger", level=3, res1=2048, res2=2048, upscale=1, depth=6,
             planes=8, map_w=2048, map_h=2048, accum="i32", hitter="bvh", material="cauchy"),
        # a moving water surface: 80,000 triangles uploaded and rebuilt every frame
        dict(name="animated_ripples", kind="animated", level=200, res1=1024, res2=1024, upscale=1, depth=2,
             planes=8, map_w=512, map_h=512, accum="i32", hitter="bvh", material="cauchy"),
        # a whole frame of the real-time scene: forward step and a 720p camera pass
        dict(name="render_720p", kind="render", scene="displaced", level=6, res1=2048, res2=2048, upscale=2, depth=4,
             planes=16, map_w=1024, map_h=1024, accum="i32", hitter="bvh", material="cauchy", height=720, width=1280),
        # a caller's own scattered rays against a resident scene, distances wanted too
        dict(name="hits_scattered", kind="hits", scene="menger", level=3, rays=120011, pencil=False, hitter="bvh"),
        # the reference's hitter over its own n_tris array
        dict(name="hits_ntris", kind="ntris", scene="sphere", level=4, rays=40000, pencil=True),
        # a Julia caller's frame: the drop-in sequence on ADRay records, float map as in the reference
        dict(name="dropin_frame", kind="dropin", scene="displaced", level=5, res1=1024, res2=1024, upscale=2, depth=4,
             planes=12, map_w=512, map_h=512, accum="f32", hitter="bvh", material="linear"),
        # the same with the bounce loop on the caller's side
        dict(name="dropin_steps", kind="steps", scene="menger", level=2, res1=700, res2=500, upscale=1, depth=3,
             planes=6, map_w=640, map_h=480, accum="i32", hitter="bvh", material="sellmeier"),
        # the backward half on caller-owned records, an odd image size
        dict(name="dropin_camera", kind="camera", scene="displaced", level=5, upscale=2, depth=4, planes=8, map_w=512,
             map_h=512, hitter="bvh", material="cauchy", height=362, width=642),
        # eight uneven frames of eight scenes, two captured engines replayed side by side
        dict(name="batch_uneven", kind="batch", frames=8, lanes=2, pick=3),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


_KINDS = ("frame", "frame", "frame", "frame", "animated", "render", "hits", "ntris", "dropin", "steps", "camera",
          "batch")


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones among them."""
    kind = rng.choice(_KINDS)
    scene = rng.choice(("sphere", "displaced", "menger"))
    level = rng.randint(1, 3) if scene == "menger" else rng.randint(2, 6)
    up = rng.choice((1, 1, 2))
    rays = _log(rng, 1 << 12, 1 << 21)
    aspect = _log(rng, 0.5, 2.0)
    res1 = max(32, int(math.sqrt(rays * aspect))) * up + rng.randrange(up)
    res2 = max(32, int(math.sqrt(rays / aspect))) * up + rng.randrange(up)
    side = int(_log(rng, 64, 1536))
    frame = dict(scene=scene, level=level, res1=res1, res2=res2, upscale=up, depth=rng.randint(2, 6),
                 planes=rng.randint(1, 16), map_w=side + rng.randint(0, 32), map_h=side,
                 accum=rng.choice(("i32", "i32", "f32")), hitter="bvh",
                 material=rng.choice(("cauchy", "cauchy", "linear", "sellmeier")))
    if kind == "frame":
        # brute force is for small frames: as in the listed ones, at most about 2^31 pairs a bounce
        if rays * _n_glass(scene, level) < 2.0 ** 30 and rng.random() < 0.5:
            frame["hitter"] = "brute"
        if rng.random() < 0.2:
            frame["planes"] = 0
        return dict(kind=kind, **frame)
    if kind == "animated":
        frame.pop("scene")
        frame["level"] = rng.randint(40, 200)
        frame["depth"] = 2
        return dict(kind=kind, **frame)
    image = dict(height=int(_log(rng, 90, 1080)) // 2 * 2, width=int(_log(rng, 160, 1920)) // 2 * 2)
    if kind == "render":
        frame.update(scene="displaced" if scene == "menger" else scene, level=rng.randint(3, 6))
        return dict(kind=kind, **frame, **image)
    if kind == "hits":
        return dict(kind=kind, scene=scene, level=level, rays=int(_log(rng, 1 << 12, 1 << 20)) | 1,
                    pencil=rng.random() < 0.5, hitter=rng.choice(("bvh", "bvh", "bvh2")))
    if kind == "ntris":
        level = rng.randint(1, 2) if scene == "menger" else rng.randint(2, 4)
        return dict(kind=kind, scene=scene, level=level, rays=int(_log(rng, 1 << 11, 1 << 17)) | 1,
                    pencil=rng.random() < 0.5)
    if kind in ("dropin", "steps"):
        # ray records are 136 bytes: such callers stay at a million rays or so
        frame.update(res1=max(32 * up, res1 // 2), res2=res2)
        return dict(kind=kind, **frame)
    if kind == "camera":
        return dict(kind=kind, scene="displaced" if scene == "menger" else scene, level=rng.randint(3, 6), upscale=2,
                    depth=frame["depth"], planes=frame["planes"], map_w=frame["map_w"], map_h=frame["map_h"],
                    hitter="bvh", material=frame["material"], **image)
    return dict(kind="batch", frames=rng.randint(2, 12), lanes=rng.randint(1, 2), pick=rng.randrange(1 << 20))


# ---------------------------------------------------------------------------
# scenes and workloads
# ---------------------------------------------------------------------------

_MATERIALS = {
    "linear": (T.MATERIAL_LINEAR_REF, 0.0, 0.0),
    "cauchy": S.CAUCHY_GLASS,
    # BK7's coefficients (micrometres)
    "sellmeier": (T.MATERIAL_SELLMEIER, 0.0, 0.0, (1.03961212, 0.231792344, 1.01046945),
                  (0.00600069867, 0.0200179144, 103.560653)),
}


def _n_glass(scene, level):
    return 12 * 20 ** level if scene == "menger" else 20 * 4 ** level


@functools.lru_cache(maxsize=None)
def _mesh(scene, level):
    """The glass of a scene before its rotation: fixed geometry, built once."""
    if scene == "menger":
        return S.menger_tris(level, 2.0, None)
    return S.sphere_tris(level, noise_amp=0.05 if scene == "displaced" else 0.0, noise_seed=3)


def _scene_tris(scene, level, seed):
    """Glass rotated by the seed, over the diffuse floor or inside the diffuse box."""
    glass = S.rotate(_mesh(scene, level), S.random_quaternion_matrix(seed + 17))
    return S.assemble(glass, S.box_tris(3.0) if scene == "menger" else S.floor_tris(-1.5, 4.0))


def _light(scene, res1, res2, seed):
    if scene == "menger":
        # from above, tilted by a few degrees
        a, b = np.random.default_rng(seed).uniform(-0.06, 0.06, 2)
        d = np.array([a, -1.0, b]) / math.sqrt(1.0 + a * a + b * b)
        d1 = np.cross(d, (0.0, 0.0, 1.0))
        d1 /= np.linalg.norm(d1)
        return T.rect_light((0.0, 2.6, 0.0), d, 1.3 * d1, 1.3 * np.cross(d, d1), res1, res2)
    light = S.hemisphere_light(seed, res1, 1.1)
    light["res2"] = res2
    return light


def _workload(c, seed, tris=None, first_diffuse=0, light=None):
    scene = c.get("scene", "")
    if tris is None:
        tris, first_diffuse = _scene_tris(scene, c["level"], seed)
        light = _light(scene, c["res1"], c["res2"], seed)
    planes = c["planes"]
    mode = (T.LAMBDA_STRATIFIED, planes, 400.0, 700.0) if planes else (T.LAMBDA_UNIFORM, 1, 400.0, 700.0)
    return S.Workload(name=c["kind"], tris=tris, first_diffuse=first_diffuse, light=light, upscale=c["upscale"],
                      lambda_mode=mode, spectrum=S.stratified_spectrum(planes) if planes else None, depth=c["depth"],
                      material=_MATERIALS[c["material"]], map_w=c["map_w"], map_h=c["map_h"], accum=c["accum"],
                      hitter=c["hitter"], seed=seed + 1)


_HITTERS = {"bvh": tracer.BVH, "bvh2": tracer.BVH2, "brute": tracer.BRUTE}


def _records(n, pencil, half, seed):
    """n active ADRay records in or around a scene of the given half extent:
    a narrow pencil through a grid, in its order, or scattered origins and
    directions."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if pencil:
        side = max(1, int(math.sqrt(n)))
        k = torch.arange(n, device="cuda")
        u = (k % side).float() / side * 2.2 - 1.1
        v = torch.div(k, side, rounding_mode="floor").float() / max(1.0, n / side) * 2.2 - 1.1
        jit = (torch.rand(n, 2, device="cuda", generator=g) - 0.5) * (2.2 / side)
        pos = torch.stack([u + jit[:, 0], torch.full_like(u, 0.9 * half), v + jit[:, 1]], 1)
        d = torch.tensor([0.05, -1.0, 0.02], device="cuda") + 0.02 * torch.randn(n, 3, device="cuda", generator=g)
    else:
        pos = (torch.rand(n, 3, device="cuda", generator=g) * 2 - 1) * (0.9 * half)
        d = torch.randn(n, 3, device="cuda", generator=g)
    d = d / d.norm(dim=1, keepdim=True)
    w = torch.zeros(n, 34, dtype=torch.float32, device="cuda")
    w[:, 0:3] = pos
    w[:, 12:15] = d
    w[:, 30] = 550.0
    i = w.view(torch.int32)
    i[:, 26] = 1  # ignore_tri: the sentinel, as a fresh ray has it
    i[:, 33] = T.STATUS_ACTIVE
    return w.view(torch.uint8).reshape(-1)


def _half(scene):
    return 3.0 if scene == "menger" else 1.4


def _batch_frames(c, seed):
    """Frames of uneven size, as the batched workload draws them; the sizes
    belong to the case, the geometry's rotation and the draws to the seed."""
    rng = np.random.default_rng(c["pick"])
    out = []
    for i in range(c["frames"]):
        scene = "menger" if rng.uniform() < 0.5 else "displaced"
        level = int(rng.integers(1, 4)) if scene == "menger" else int(rng.integers(3, 6))
        res = max(128, int(math.sqrt(math.exp(rng.uniform(math.log(2 ** 14), math.log(2 ** 19))))))
        side = int(math.exp(rng.uniform(math.log(256), math.log(1024))))
        out.append(dict(kind="batch", scene=scene, level=level, res1=res, res2=res, upscale=1,
                        depth=int(rng.integers(2, 7)), planes=int(rng.integers(1, 13)), map_w=side, map_h=side,
                        accum="i32", hitter="bvh", material="cauchy"))
    return out


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"case": c}
    if kind == "frame":
        st["step"] = tracer.TraceStep(_workload(c, seed))
    elif kind == "animated":
        n = c["level"]
        t = 0.25 + (seed % 1000) * 0.01
        rips = S.translate(S.ripples(t, 1.0 / n), (-0.5, -0.5, 0.0))
        tris, fd = S.assemble_meshes([rips], [S.translate(S.square(), (-0.5, -1.0, -3.0))])
        light = T.rect_light((0.0, 0.0, 2.0), (0.0, 0.0, -1.0), (0.6, 0.0, 0.0), (0.0, 0.6, 0.0), c["res1"], c["res2"])
        st["step"] = tracer.TraceStep(_workload(c, seed, tris, fd, light))
        st["tris"] = torch.from_numpy(tris).cuda()
        st["step"].scene.rebuild(st["tris"])  # the first rebuild allocates its scratch
    elif kind == "render":
        wl = _workload(c, seed)
        cam = S.realtime_camera()
        view = tracer.camera_look_at(cam["pos"], cam["look_at"], cam["up"], cam["fov"])
        sky = torch.from_numpy(np.ascontiguousarray(S.gradient_sky().transpose(2, 1, 0))).cuda()
        st["renderer"] = tracer.Renderer(wl, view, c["height"], c["width"], sky=sky)
    elif kind in ("hits", "ntris"):
        tris, fd = _scene_tris(c["scene"], c["level"], seed)
        st["rays"] = _records(c["rays"], c["pencil"], _half(c["scene"]), seed)
        if kind == "hits":
            st["scene"] = tracer.Scene(tris, fd)
        else:
            st["ntris"] = tracer.n_tris_array(tris)
    elif kind in ("dropin", "steps"):
        wl = _workload(c, seed)
        st.update(wl=wl, scene=tracer.Scene(wl.tris, wl.first_diffuse), spectrum=wl.spectrum,
                  tex=tracer.new_light_map(wl.map_w, wl.map_h, wl.n_planes, wl.accum))
        n = wl.n_rays
        lib = tracer.L.load()
        if kind == "dropin":
            st["ws"] = torch.empty(int(lib.splat_run_evolution_workspace_size(n)), dtype=torch.uint8, device="cuda")
        else:
            st["ws"] = torch.empty(int(lib.splat_partition_workspace_size(n)), dtype=torch.uint8, device="cuda")
    elif kind == "camera":
        tris, fd = _scene_tris(c["scene"], c["level"], seed)
        cam = S.realtime_camera()
        st.update(scene=tracer.Scene(tris, fd), seed=seed + 1, spectrum=S.stratified_spectrum(c["planes"]),
                  cam=tracer.camera_look_at(cam["pos"], cam["look_at"], cam["up"], cam["fov"]))
        st["retina"] = tracer.retina_factors(st["spectrum"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["map"] = torch.rand((c["planes"], c["map_h"], c["map_w"]), device="cuda", generator=g)
        st["shader"] = tracer.Shader(c["map_w"], c["map_h"], c["planes"], 512, 256)
        st["shader"].set_skydome(torch.from_numpy(np.ascontiguousarray(S.gradient_sky().transpose(2, 1, 0))).cuda())
        n = (c["height"] // c["upscale"]) * (c["width"] // c["upscale"])
        st["ws"] = torch.empty(int(tracer.L.load().splat_run_evolution_workspace_size(n)), dtype=torch.uint8,
                               device="cuda")
        st["rgb"] = tracer.new_image(c["height"], c["width"])
    else:
        frames = [_workload(f, seed + i) for i, f in enumerate(_batch_frames(c, seed))]
        st["scenes"] = [tracer.Scene(w.tris, w.first_diffuse) for w in frames]
        st["maps"] = [tracer.new_light_map(w.map_w, w.map_h, w.n_planes, w.accum) for w in frames]
        st["lanes"] = batch.Lanes(c["lanes"], frames, st["scenes"], st["maps"])
        st["lanes"].capture()
        st["seeds"] = [w.seed for w in frames]
    return st


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "frame":
        step = state["step"]
        return {"map": step.run(), "counts": step.d_stats}
    if kind == "animated":
        step = state["step"]
        step.scene.rebuild(state["tris"])
        return {"map": step.run(), "counts": step.d_stats}
    if kind == "render":
        r = state["renderer"]
        return {"image": r.run(), "map": r.step.tex}
    if kind == "hits":
        hit, t = tracer.next_hit(state["scene"], _HITTERS[c["hitter"]], state["rays"], with_t=True)
        return {"hit": hit, "t": t}
    if kind == "ntris":
        hit, packed = tracer.next_hit_brute(state["rays"], state["ntris"])
        return {"hit": hit, "packed": packed}
    if kind == "dropin":
        wl, tex = state["wl"], state["tex"]
        tex.zero_()
        rays = tracer.rays_from_light(wl.light, wl.upscale, wl.lambda_mode, wl.seed)
        hit = tracer.run_evolution(_HITTERS[c["hitter"]], state["scene"], rays, wl.depth, wl.material, None, wl.seed,
                                   wl.quirks, state["ws"])
        tracer.continuum_light_map2(state["scene"], rays, hit, state["spectrum"], wl.upscale, tex, wl.frac_bits)
        return {"map": tex, "rays": rays, "hit": hit}
    if kind == "steps":
        wl, tex, scene = state["wl"], state["tex"], state["scene"]
        hitter = _HITTERS[c["hitter"]]
        tex.zero_()
        rays = tracer.rays_from_light(wl.light, wl.upscale, wl.lambda_mode, wl.seed)
        live, counts = rays, []
        for b in range(1, wl.depth + 1):
            hit = tracer.next_hit(scene, hitter, live)
            # one draw for all: the rays' order after a partition is free
            tracer.evolve(scene, live, hit, wl.material, None, 0.5, wl.seed, b, wl.quirks)
            n = int(tracer.partition(live, state["ws"]).item())  # the reference reads the count back too
            counts.append(n)
            if n == 0:
                break
            live = live[: n * T.ADRAY.itemsize]
        hit = tracer.next_hit(scene, hitter, rays)
        tracer.continuum_light_map2(scene, rays, hit, state["spectrum"], wl.upscale, tex, wl.frac_bits)
        return {"map": tex, "counts": counts}
    if kind == "camera":
        sh, up = state["shader"], c["upscale"]
        sh.set_light_map(state["map"])
        rays = tracer.camera_rays(state["cam"], c["height"] // up, c["width"] // up, 550.0, state["seed"])
        hit = tracer.run_evolution(_HITTERS[c["hitter"]], state["scene"], rays, c["depth"], _MATERIALS[c["material"]],
                                   None, state["seed"], True, state["ws"])
        rgb = tracer.continuum_shade(state["scene"], sh, rays, hit, state["spectrum"], state["retina"], up,
                                     c["height"], c["width"], state["rgb"])
        return {"image": rgb, "rays": rays, "hit": hit}
    state["lanes"].replay(state["seeds"])
    return {"maps": state["maps"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

_ADRAY = 136
_TRI = 120


def _n_tris(c):
    if c["kind"] == "animated":
        return 2 * c["level"] ** 2 + 3
    return _n_glass(c["scene"], c["level"]) + (13 if c["scene"] == "menger" else 3)


def _trace_flops(n_rays, n_tris, depth, hitter, samples):
    """Ray segments times a hit search and an evolve, and the splat samples.
    A segment's rays: all of them on the first bounce, about two thirds on
    each later one.  A search: 30 operations a plane-and-edges test of every
    triangle, or 4 boxes of 12 operations a level of a four-wide tree."""
    segments = n_rays * (1.0 + 0.65 * (depth - 1))
    search = 30.0 * n_tris if hitter == "brute" else 48.0 * max(1.0, math.log(n_tris, 4))
    return segments * (search + 600.0) + 0.6 * n_rays * samples * 100.0


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        parts = [work(dict(f, kind="frame")) for f in _batch_frames(c, 0)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    n_tris = _n_tris(c)
    if kind in ("hits", "ntris"):
        # origin, direction, triangle to ignore in; index and distance out
        flops = _trace_flops(c["rays"], n_tris, 1, "brute" if kind == "ntris" else c["hitter"], 0) - 600.0 * c["rays"]
        return {"bytes": c["rays"] * (28 + 8) + n_tris * 52, "flops": flops}
    if kind == "camera":
        n = (c["height"] // c["upscale"]) * (c["width"] // c["upscale"])
        texels = c["map_w"] * c["map_h"] * c["planes"]
        return {"bytes": n * (_ADRAY + 4) + texels * 4 + c["height"] * c["width"] * 12 + n_tris * _TRI,
                "flops": _trace_flops(n, n_tris, c["depth"], c["hitter"], c["planes"] * c["upscale"] ** 2)}
    n = (c["res1"] // c["upscale"]) * (c["res2"] // c["upscale"])
    planes = max(1, c["planes"])
    bytes_ = c["map_w"] * c["map_h"] * planes * 4 + n_tris * _TRI
    flops = _trace_flops(n, n_tris, c["depth"], c["hitter"], planes * c["upscale"] ** 2)
    if kind in ("dropin", "steps"):
        bytes_ += n * (_ADRAY + 4)
    if kind == "animated":
        bytes_ += n_tris * (_TRI + 80)
    if kind == "render":
        cam = (c["height"] // 2) * (c["width"] // 2)
        bytes_ += c["height"] * c["width"] * 12
        flops += _trace_flops(cam, n_tris, c["depth"], c["hitter"], planes * 4)
    return {"bytes": float(bytes_), "flops": float(flops)}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------


def exact(case, seed):
    """The hit distances, by a search over every triangle in 64 bits.

    The other cases have no such value: their integer maps, records and
    indices are whole numbers, and a float map or an image sums samples whose
    triangle, Fresnel branch and texel are picked by 32-bit comparisons (the
    image also through the texture unit's 8-bit filter weights)."""
    c = case
    if c["kind"] != "hits" or c["rays"] * _n_tris(c) > 1.2e10:
        return None
    tris, _ = _scene_tris(c["scene"], c["level"], seed)
    rays = _records(c["rays"], c["pencil"], _half(c["scene"]), seed).view(torch.float32).view(-1, 34)
    o, d = rays[:, 0:3].double(), rays[:, 12:15].double()
    f = torch.from_numpy(tris[1:]).cuda().double()
    n, a, e0, e1 = f[:, 0], f[:, 1], f[:, 3] - f[:, 1], f[:, 2] - f[:, 1]
    d00, d01, d11 = (e0 * e0).sum(1), (e0 * e1).sum(1), (e1 * e1).sum(1)
    inv = 1.0 / (d00 * d11 - d01 * d01)
    # u = p . A + a0 and v = p . B + b0 on the triangle's plane
    A = (e0 * d11[:, None] - e1 * d01[:, None]) * inv[:, None]
    B = (e1 * d00[:, None] - e0 * d01[:, None]) * inv[:, None]
    a0, b0, nv = (A * a).sum(1), (B * a).sum(1), (n * a).sum(1)
    best = torch.full((c["rays"],), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, int(1.0e8) // c["rays"])
    for j in range(0, n.shape[0], step):
        s = slice(j, j + step)
        t = (nv[s] - o @ n[s].T) / (d @ n[s].T)
        u = (o @ A[s].T - a0[s]).addcmul_(d @ A[s].T, t)
        v = (o @ B[s].T - b0[s]).addcmul_(d @ B[s].T, t)
        ok = (t > 0) & (u >= 0) & (v >= 0) & (u + v < 1)
        best = torch.minimum(best, torch.where(ok, t, math.inf).amin(1))
    return {"hit": None, "t": best}
