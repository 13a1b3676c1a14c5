"""The work a user of this renderer has it do, as measurable cases.

A case is a dict of plain values. `op` says which public entry point it goes
through (`Renderer.render` for a frame, a crop, a capture or the plain
megakernel; `rt_render_batch` for many requests in one launch;
`adjoint.render_function` for a forward + backward step of a fit;
`Renderer.tone_map_to_display` for showing a film again at another exposure),
`scene` which of the package's scenes it renders, the rest the sizes and
options. `prepare` builds what a program holds before the call (the scene on
the GPU, the requests, the target image); `run` is one call.

Every input comes from the seed: it moves the camera, changes the materials'
colours and roughnesses (the icosphere field is another field altogether) and
picks the Sobol range that is rendered.

Rendered films have no 64-bit counterpart: a path's decisions (which triangle,
which lobe, when roulette ends it) are made on its own 32-bit numbers, so the
same paths in 64 bits are other paths. `exact` gives a value for the display
transform alone.
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package lives in 3d-ray_b200/ (not an identifier): load it as rt3d_b200."""
    if "rt3d_b200" not in sys.modules:
        d = os.path.join(_ROOT, "3d-ray_b200")
        spec = importlib.util.spec_from_file_location("rt3d_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        m = importlib.util.module_from_spec(spec)
        sys.modules["rt3d_b200"] = m
        spec.loader.exec_module(m)
    return sys.modules["rt3d_b200"]


# --- the cases ----------------------------------------------------------------

def listed():
    return [
        # A thumbnail or the first pass of an interactive view: the smallest call, all latency.
        dict(name="preview_thumbnail", op="render", scene="cornell", width=64, height=48, spp=4, depth=4),
        # The Cornell box at its usual size, depth and sample count: an ordinary still.
        dict(name="cornell_still", op="render", scene="cornell", width=256, height=256, spp=64, depth=8),
        # A full-HD frame of the 1.3 M triangle icosphere field, the largest render.
        dict(name="icospheres_full_hd", op="render", scene="icospheres", spheres=64, level=5, width=1920, height=1080,
             spp=64, depth=12),
        # A progressive pass over a ragged crop of a frame (the user drags a render region): few samples
        # of odd sizes into a mid-sized scene.
        dict(name="icospheres_crop_pass", op="render", scene="icospheres", spheres=33, level=4, width=1277, height=719,
             spp=8, depth=10, x0=211, y0=101, window_w=517, window_h=333),
        # An open scene under a sky with glass, light picking by power and the power heuristic: transparent
        # shadows, the IOR stack, sky misses.
        dict(name="sky_glass_still", op="render", scene="sky", width=641, height=361, spp=48, depth=10, lights="power",
             mis="power"),
        # Smooth meshes, an emissive mesh and an anisotropic metal: interpolated normals and mesh lights.
        dict(name="smooth_mesh_still", op="render", scene="smooth", width=400, height=300, spp=32, depth=8),
        # A render farm's batch: uneven requests over two scenes in one launch.
        dict(name="mixed_batch", op="batch", scene="mixed", spheres=64, level=4, requests=12, lo=64, hi=512, spp_lo=16,
             spp_hi=128),
        # Views of a foggy box with a dielectric sphere in one launch: a medium, NEE inside it, absorption.
        dict(name="volume_views", op="batch", scene="volume", requests=4, lo=256, hi=256, spp_lo=64, spp_hi=64),
        # A render with the denoiser's side buffers: sample halves, albedo, normal and depth.
        dict(name="denoiser_capture", op="capture", scene="icospheres", spheres=24, level=3, width=321, height=243,
             spp=16, depth=8),
        # One step of fitting a sphere's material and the light to an image: forward, then the adjoint.
        dict(name="material_fit_step", op="fit", scene="sphere", width=256, height=256, spp=32, depth=8),
        # One step of fitting the fog (absorption and scattering): the adjoint through a medium.
        dict(name="medium_fit_step", op="fit", scene="volume", width=64, height=64, spp=128, depth=16),
        # An exposure slider on a finished full-HD film: the display transform alone.
        dict(name="re_expose_full_hd", op="display", scene="film", width=1920, height=1080, ev=0.75),
    ]


# Nanoseconds a sample of a scene costs at the start, roughly; they only keep drawn cases affordable.
_NS = dict(cornell=4.0, sphere=4.0, smooth=8.0, spheres=10.0, sky=6.0, icospheres=1.6, volume=7.0)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["render"] * 6 + ["batch"] * 2 + ["capture", "megakernel", "fit", "fit", "display"])
    if op == "display":
        return dict(op=op, scene="film", width=_log(rng, 31, 3840), height=_log(rng, 17, 2160),
                    ev=round(rng.uniform(-3.0, 3.0), 3))
    if op == "batch":
        hi = _log(rng, 96, 384)
        return dict(op=op, scene=rng.choice(["mixed", "mixed", "volume"]), spheres=rng.randint(4, 48),
                    level=rng.randint(2, 4), requests=rng.randint(2, 10), lo=_log(rng, 24, 96), hi=hi,
                    spp_lo=rng.randint(1, 8), spp_hi=_log(rng, 9, 64))
    if op == "fit":
        scene = rng.choice(["sphere", "sphere", "volume"])
        side = _log(rng, 24, 160 if scene == "sphere" else 72)
        return dict(op=op, scene=scene, width=side, height=side + rng.randint(-7, 7), spp=_log(rng, 2, 48),
                    depth=rng.randint(4, 12))
    scene = rng.choice(["cornell", "sphere", "smooth", "spheres", "sky", "volume", "icospheres", "icospheres"])
    c = dict(op="render" if op == "megakernel" else op, scene=scene, width=_log(rng, 40, 1920), depth=rng.randint(2, 14))
    c["height"] = max(16, int(c["width"] * rng.uniform(0.5, 1.1)))
    if scene == "icospheres":
        c.update(spheres=rng.randint(1, 64), level=rng.randint(1, 4))
    if op == "megakernel":
        c["kernel"] = "megakernel"
    budget_ms = 0.5 * 64 * 1920 * 1080 * _NS["icospheres"] / 1e6
    ns = _NS[scene] * (8.0 if op != "render" else 1.0)
    if op != "render":   # the plain kernel renders small images in practice
        c["width"], c["height"] = min(c["width"], 320), min(c["height"], 240)
    most = max(1, min(96, int(budget_ms * 1e6 / (ns * c["width"] * c["height"]))))
    c["spp"] = _log(rng, 1, most)
    if op == "render":
        if rng.random() < 0.3:
            c.update(lights=rng.choice(["power", "uniform"]), mis=rng.choice(["balance", "power"]))
        if rng.random() < 0.3:
            c["x0"], c["y0"] = rng.randint(0, c["width"] // 3), rng.randint(0, c["height"] // 3)
            c["window_w"] = rng.randint(8, c["width"] - c["x0"])
            c["window_h"] = rng.randint(8, c["height"] - c["y0"])
    return c


# --- inputs -------------------------------------------------------------------

def _world(rt, case, scene, rng):
    """The named scene, with the seed's camera and materials."""
    sc = rt.scenes
    if scene == "icospheres":
        w = sc.throughput_scene(seed=int(rng.integers(1 << 20)), n_spheres=case["spheres"], level=case["level"])
    else:
        w = {"cornell": sc.cornell, "sphere": sc.cornell_sphere, "smooth": sc.cornell_smooth,
             "spheres": sc.cornell_spheres, "sky": sc.sky_scene, "volume": sc.cornell_volume}[scene]()
        for m in w.materials:
            if m["type"] == 0:
                m["base_color"] = tuple(float(np.clip(c * rng.uniform(0.7, 1.3), 0.02, 0.95)) for c in m["base_color"])
                if m["roughness"] > 0.1:
                    m["roughness"] = float(np.clip(m["roughness"] * rng.uniform(0.7, 1.0), 0.1, 1.0))
    cam = w.camera
    eye, at = np.array(cam["look_from"]), np.array(cam["look_at"])
    w.camera = sc.camera(tuple(eye + 0.03 * np.linalg.norm(at - eye) * rng.uniform(-1, 1, 3) * (1, 1, 0)), tuple(at),
                         cam["vup"], cam["vfov"], cam["aperture"], cam["focus_dist"])
    return w


def _request_sizes(case):
    """(scene, width, height, spp) of a batch's requests: sides and sample counts spread over the case's
    ranges (their logarithms), large images with few samples and the other way round."""
    n = case["requests"]
    spread = lambda k, lo, hi: int(round(lo * (hi / lo) ** (((k * 5) % n) / max(1, n - 1))))  # noqa: E731
    for k in range(n):
        side, spp = spread(k, case["lo"], case["hi"]), spread(n - 1 - k, case["spp_lo"], case["spp_hi"])
        yield (0, side, side, spp) if case["scene"] == "volume" else (k % 2, side, side + k % 3, spp)


def _requests(rt, case, rng):
    """Uneven requests: the mixed batch over scenes 0 (icospheres) and 1 (Cornell box) from cameras around
    them, the volume batch from the box's open side."""
    sc = rt.scenes
    views = sc.volume_views(8)
    reqs = []
    for k, (scene, width, height, spp) in enumerate(_request_sizes(case)):
        if case["scene"] == "volume":
            reqs.append(dict(scene=0, width=width, height=height, spp=spp, max_depth=16,
                             camera=views[(k + int(rng.integers(8))) % 8]))
            continue
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        if scene == 1:
            d[2] = -abs(d[2]) - 0.5
            center, r = np.array([278.0, 278.0, 278.0]), 1000.0
        else:
            d[1] = abs(d[1]) * 0.6 + 0.1
            center, r = np.array([0.0, -1.0, 0.0]), 25.0
        d /= np.linalg.norm(d)
        reqs.append(dict(scene=scene, width=width, height=height, spp=spp, max_depth=4 + k % 9,
                         camera=sc.camera(tuple(center + d * r), tuple(center), (0, 1, 0), 40.0)))
    return reqs


def prepare(case, seed):
    rt = _package()
    rng = np.random.default_rng([int(seed), 77])
    op = case["op"]
    if op == "display":
        # HDR radiances: mostly of order one, a few far brighter, some black pixels
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        film = torch.randn((3, case["height"], case["width"]), generator=g, device="cuda")
        film = torch.exp(1.5 * film - 1.0)
        film *= (torch.rand((1, case["height"], case["width"]), generator=g, device="cuda") > 0.1)
        r = rt.renderer.Renderer(rt.scenes.cornell(), 1, 1, exposure_ev=case["ev"])
        return dict(op=op, renderer=r, film=film.cpu().numpy())
    if op == "batch":
        kinds = ["volume"] if case["scene"] == "volume" else ["icospheres", "cornell"]
        scenes = [rt.renderer.Renderer(_world(rt, case, k, rng), 1, 1) for k in kinds]
        reqs = _requests(rt, case, rng)
        arr = (rt.abi.RtRequest * len(reqs))()
        for q, r in zip(arr, reqs):
            q.scene, q.width, q.height, q.spp, q.max_depth = (r[k] for k in ("scene", "width", "height", "spp", "max_depth"))
            q.camera = rt.abi.camera_desc(r["camera"])
        return dict(op=op, rt=rt, scenes=scenes, reqs=arr, handles=(C.c_void_p * len(scenes))(*[s._scene.value for s in scenes]),
                    common=rt.abi.render_params(1, 1, 1, 1, kernel=rt.abi.KERNEL_WAVEFRONT))
    w = _world(rt, case, case["scene"], rng)
    offset = int(rng.integers(4096))
    if op == "fit":
        d = rt.adjoint.DiffScene(w)
        params = rt.abi.render_params(case["width"], case["height"], case["spp"], case["depth"],
                                      kernel=rt.abi.KERNEL_WAVEFRONT, spp_offset=offset)
        theta = d.get_params()
        if case["scene"] == "volume":
            slots = [d.medium_slot(k, c) for k in ("sigma_a", "sigma_s") for c in range(3)]
        else:
            slots = [d.slot("fit_sphere", "base_color", c) for c in range(3)]
            slots += [d.slot("fit_sphere", k) for k in ("roughness", "metallic", "specular", "sheen")]
            slots += [d.slot("light", "radiance", c) for c in range(3)]
            theta[slots[3:7]] = rng.uniform(0.2, 0.8, 4)
        target = rng.uniform(0.0, 0.6, (3, case["height"], case["width"])).astype(np.float32)
        return dict(op=op, scene=d, params=params, slots=slots, fn=rt.adjoint.render_function(),
                    theta=torch.from_numpy(theta).requires_grad_(True), target=torch.from_numpy(target))
    r = rt.renderer.Renderer(w, case["spp"], case["depth"], mis_heuristic=case.get("mis", "balance"),
                             light_sampling_strategy=case.get("lights", "all"), kernel=case.get("kernel", "wavefront"))
    kw = dict(spp_offset=offset)
    if "window_w" in case:
        kw.update(pixel_x0=case["x0"], pixel_y0=case["y0"], window_w=case["window_w"], window_h=case["window_h"])
    cap = rt.renderer.RenderCaptureOptions.FULL if op == "capture" else None
    return dict(op=op, renderer=r, size=(case["width"], case["height"]), kw=kw, capture=cap)


# --- one pass -----------------------------------------------------------------

def run(state):
    op = state["op"]
    if op == "display":
        return state["renderer"].tone_map_to_display(state["film"])
    if op == "batch":
        rt, reqs = state["rt"], state["reqs"]
        outs = [np.zeros((3, q.height, q.width), np.float32) for q in reqs]
        ptrs = (C.c_void_p * len(outs))(*[o.ctypes.data for o in outs])
        st = rt.abi.RtStats()
        rt.abi.check(rt.abi.load().rt_render_batch(state["handles"], len(state["handles"]), reqs, len(outs),
                                                   C.byref(state["common"]), ptrs, C.byref(st)), "rt_render_batch")
        return outs
    if op == "fit":
        theta = state["theta"]
        theta.grad = None
        image = state["fn"].apply(theta, state["scene"], state["params"], state["slots"])
        loss = ((image - state["target"]) ** 2).mean()
        loss.backward()
        return dict(image=image.detach(), grad=theta.grad)
    r = state["renderer"].render(*state["size"], capture=state["capture"], **state["kw"])
    out = dict(pixels=r.pixels, beauty=r.beauty)
    if r.buffers is not None:
        for k in ("beauty_a", "beauty_b", "albedo_a", "albedo_b", "normal_a", "normal_b", "depth_a", "depth_b"):
            out[k] = getattr(r.buffers, k)
    return out


# --- what a pass cannot do without ------------------------------------------------

# Per camera sample at the scene's usual depth: the box, triangle and quad / sphere tests of its closest
# and shadow rays, as the counting build counts the reference's walk, and the vertices it shades. A box
# test is 24 operations, a triangle 60, a quad or sphere 40, a vertex (light samples, BSDF sample, value
# and density, roulette) about 900.
_PER_SAMPLE = dict(cornell=(46.2, 13.1, 23.8, 3.5), sphere=(56.6, 12.3, 23.4, 3.6), smooth=(90.3, 17.0, 28.8, 3.5),
                   spheres=(115.4, 15.0, 131.9, 3.5), sky=(0.0, 0.0, 11.2, 1.2), volume=(66.0, 4.0, 54.1, 6.2),
                   icospheres=(85.1, 8.4, 0.4, 0.5))


def _flops(scene, samples):
    box, tri, other, vert = _PER_SAMPLE[scene]
    return samples * (24.0 * box + 60.0 * tri + 40.0 * other + 900.0 * vert)


def _scene_bytes(case, scene):
    """Triangles (9 floats) and their tree (one 32 B box for every two), read once."""
    if scene != "icospheres":
        return 64e3 if scene == "smooth" else 4e3
    return case["spheres"] * 20 * 4 ** case["level"] * (36 + 16)


def work(case):
    op, scene = case["op"], case["scene"]
    if op == "display":
        n = 3 * case["width"] * case["height"]
        return dict(bytes=8.0 * n, flops=30.0 * n)
    if op == "batch":
        b = f = 0.0
        kinds = ["volume"] if scene == "volume" else ["icospheres", "cornell"]
        for k, width, height, spp in _request_sizes(case):
            b += 12.0 * width * height
            f += _flops(kinds[k], width * height * spp)
        return dict(bytes=b + sum(_scene_bytes(case, k) for k in kinds), flops=f)
    px = case.get("window_w", case["width"]) * case.get("window_h", case["height"])
    full = case["width"] * case["height"]
    f = _flops(scene, px * case["spp"])
    planes = dict(render=6, capture=6 + 20, fit=6)[op]   # film and display pixels; side buffers; film and its gradient
    if op == "fit":
        f *= 4.0   # the forward film, then the adjoint: the samples again, and their replay with derivatives
    return dict(bytes=4.0 * planes * full + _scene_bytes(case, scene), flops=f)


def exact(case, seed):
    if case["op"] != "display":
        return None   # see the module's comment: other numbers take other paths
    x = np.maximum(prepare(case, seed)["film"].astype(np.float64) * float(np.float32(2.0 ** case["ev"])), 0.0)
    y = np.clip(x * (2.51 * x + 0.03) / (x * (2.43 * x + 0.59) + 0.14), 0.0, 1.0)
    return np.ascontiguousarray((y ** (1.0 / 2.2)).transpose(1, 2, 0))
