"""The wavefront and the walks at the sizes and shapes where their dispatch
changes: free-list tails of the camera kernel, chunks of the material sort, the
lines between untuned configurations, the opened-up top level for every number
and kind of entity, and the host copies' windows. Everything here runs on the
GPU, against the megakernel, the oracle or numpy."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import random_rays, rt

pytestmark = pytest.mark.gpu

abi, S = rt.abi, rt.scenes


class Scene:
    def __init__(self, world):
        self.lib, self.packed, self.h = abi.load(), abi.PackedWorld(world), C.c_void_p()
        abi.check(self.lib.rt_scene_create(self.packed.ref(), C.byref(self.h)), "rt_scene_create")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.lib.rt_scene_destroy(self.h)

    def render(self, w, h, spp, depth, **kw):
        p = abi.render_params(w, h, spp, depth, **kw)
        out, st = np.zeros((3, h, w), np.float32), abi.RtStats()
        abi.check(self.lib.rt_render(self.h, C.byref(p), abi.ptr(out), C.byref(st)), "rt_render")
        return out


def nested_glass():
    """Glass spheres inside glass spheres: IOR stacks deeper than one, interior
    absorption switched on and off, thin walls beside solid ones."""
    w = S.cornell(tall_box=False)
    for k, (r, ior, tc) in enumerate([(120.0, 1.5, (0.7, 0.9, 0.8)), (80.0, 1.2, None), (40.0, 1.7, (0.9, 0.5, 0.6))]):
        m = w.add_material(f"glass{k}", S.disney((1.0, 1.0, 1.0), roughness=0.0 if k != 1 else 0.3, spec_trans=1.0,
                                                 ior=ior, transmission_color=tc, transmission_depth=100.0))
        w.add_sphere((300, 180, 300), r, m)
    thin = w.add_material("thin", S.disney((0.9, 0.9, 1.0), roughness=0.0, spec_trans=1.0, ior=1.4, thin_walled=True))
    w.add_quad((100, 100, 150), (200, 0, 0), (0, 200, 0), thin)
    return w


WORLDS = dict(cornell=S.cornell, smooth=S.cornell_smooth, spheres=S.cornell_spheres, sky=S.sky_scene,
              volume=S.cornell_volume, glass=nested_glass,
              icospheres=lambda: S.throughput_scene(n_spheres=5, level=2))


# The same samples: a sample's terms (at most two lights at 12 vertices) differ by
# their float order, 24 x 2^-24, and the megakernel's chunk sums by one rounding a
# sample, so 1e-5 relative covers 64 samples; films are sums of positive terms.
def same_film(a, b):
    np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("world", list(WORLDS))
@pytest.mark.parametrize("w,h,spp,depth,kw", [
    (1, 1, 1, 6, {}),                                  # one sample
    (33, 7, 3, 12, {}),                                # ragged strips, fewer slots than a block
    (41, 29, 17, 8, dict(wavefront_size=1024)),        # many refills of a small free list
    (57, 43, 29, 5, dict(ray_groups=4, sort_materials=1)),
    (64, 40, 40, 2, dict(ray_groups=1, sort_materials=0)),
])
def test_small_renders_equal_the_megakernel(world, w, h, spp, depth, kw):
    with Scene(WORLDS[world]()) as s:
        ref = s.render(w, h, spp, depth, kernel=abi.KERNEL_MEGAKERNEL)
        got = s.render(w, h, spp, depth, kernel=abi.KERNEL_WAVEFRONT, **kw)
    same_film(got, ref)


# Slots around a sort chunk (65536), a regen block (512), a shade block per SM and
# the untuned configurations' lines (2^16 and 2^18 slots).
@pytest.mark.parametrize("slots", [1, 1025, 65280, 65536, 65792, 131328, (1 << 18) - 256, (1 << 18) + 256])
@pytest.mark.parametrize("world", ["icospheres", "volume"])
def test_slot_counts_render_the_same_film(world, slots):
    with Scene(WORLDS[world]()) as s:
        ref = s.render(160, 120, 16, 6, kernel=abi.KERNEL_MEGAKERNEL)
        for kw in (dict(), dict(ray_groups=4, sort_materials=1)):
            same_film(s.render(160, 120, 16, 6, kernel=abi.KERNEL_WAVEFRONT, wavefront_size=slots, **kw), ref)


# Slots around one and two turns of the shadow scatter's threads (1480 blocks of
# 256) and a shade block on every SM (148 of 512), whose next wave is prefetched.
@pytest.mark.parametrize("slots", [75776, 75776 + 256, 378880 - 256, 378880, 378880 + 256, 2 * 378880 + 256])
@pytest.mark.parametrize("world", ["icospheres", "smooth"])
def test_sorted_shadows_take_turns(world, slots):
    with Scene(WORLDS[world]()) as s:
        ref = s.render(320, 240, 16, 4, kernel=abi.KERNEL_MEGAKERNEL)
        same_film(s.render(320, 240, 16, 4, kernel=abi.KERNEL_WAVEFRONT, wavefront_size=slots, ray_groups=4,
                           sort_materials=1), ref)


def test_a_tuned_large_render_is_not_slower_than_an_untuned_one():
    """133 M samples: an untuned render of that size takes 8 M slots, which the slice
    that the autotuner's candidates run on cannot fill. The least of several device
    times each, in turn, repeats within half a percent; 4 M would be 4% slower."""
    world = S.throughput_scene()
    with Scene(world) as s, Scene(world) as plain:
        def render(scene, p):
            out, st = np.zeros((3, 1080, 1920), np.float32), abi.RtStats()
            abi.check(scene.lib.rt_render(scene.h, C.byref(p), abi.ptr(out), C.byref(st)), "rt_render")
            return out, st

        base = abi.render_params(1920, 1080, 64, 12, kernel=abi.KERNEL_WAVEFRONT)
        ref, _ = render(plain, base)
        best = abi.RtRenderParams()
        abi.check(s.lib.rt_autotune(s.h, C.byref(base), C.byref(best)), "rt_autotune")
        assert best.wavefront_size in (1 << 18, 1 << 20, 1 << 22, 1 << 23)
        runs = [(render(plain, base), render(s, base)) for _ in range(6)]
        untuned, tuned = ([r[k][1].kernel_ms for r in runs] for k in (0, 1))
        assert min(tuned) < 1.02 * min(untuned), (tuned, untuned, best.wavefront_size)
        img, st = render(s, best)   # what it returned is what it uses
        same_film(img, ref)
        same_film(runs[0][1][0], ref)
        assert abs(st.iterations - runs[0][1][1].iterations) <= 2


# Materials around the number of keys the material sort holds (256, two of them for
# what is no material): the most that sort, and one more.
@pytest.mark.parametrize("n", [253, 254, 255])
def test_material_sort_up_to_its_keys(n):
    w = S.cornell()
    while len(w.materials) < n:
        k = len(w.materials)
        m = w.add_material(f"m{k}", S.disney((0.2 + 0.7 * (k % 7) / 7, 0.5, 0.9 - 0.6 * (k % 5) / 5)))
        w.add_sphere((30.0 + 500 * (k % 16) / 16, 30.0 + 500 * (k // 16) / 16, 300.0), 14.0, m)
    with Scene(w) as s:
        ref = s.render(120, 90, 8, 4, kernel=abi.KERNEL_MEGAKERNEL)
        launches = []
        for sort in (0, 1):
            p = abi.render_params(120, 90, 8, 4, kernel=abi.KERNEL_WAVEFRONT, sort_materials=sort, ray_groups=1)
            out, st = np.zeros((3, 90, 120), np.float32), abi.RtStats()
            abi.check(s.lib.rt_render(s.h, C.byref(p), abi.ptr(out), C.byref(st)), "rt_render")
            same_film(out, ref)
            launches.append((st.kernel_launches - 1) // st.iterations)
    assert launches[1] - launches[0] == (1 if n <= 254 else 0)


# Shadow samples whose records a vertex fill one axis of a grid, and one more row.
# Film values are sums of that many positive terms in another order: each addition
# rounds by 2^-24 of the sum at most, 65 536 x 2^-24 on either side.
@pytest.mark.parametrize("side", [255, 256])
@pytest.mark.parametrize("kw", [dict(ray_groups=1), dict(ray_groups=2), dict(ray_groups=4, sort_materials=1)])
def test_a_light_of_many_shadow_samples(side, kw):
    with Scene(S.cornell(shadow_samples=side * side)) as s:
        ref = s.render(6, 5, 1, 2, kernel=abi.KERNEL_MEGAKERNEL)
        got = s.render(6, 5, 1, 2, kernel=abi.KERNEL_WAVEFRONT, **kw)
    assert ref.any()
    np.testing.assert_allclose(got, ref, rtol=2 * 65536 * 2.0 ** -24, atol=1e-6)


def large_render_in_a_full_device():
    """Run by the test below in a process of its own (its workspace starts empty)."""
    import torch
    spare = 256 << 20
    size = dict(w=1024, h=1024, spp=33, depth=2, kernel=abi.KERNEL_WAVEFRONT)   # 34.6 M samples, past the 8 M line
    with Scene(S.cornell()) as s:
        stats = abi.RtStats()

        def render(**kw):
            p = abi.render_params(size["w"], size["h"], size["spp"], size["depth"], kernel=size["kernel"], **kw)
            out = np.zeros((3, size["h"], size["w"]), np.float32)
            abi.check(s.lib.rt_render(s.h, C.byref(p), abi.ptr(out), C.byref(stats)), "rt_render")
            return out, stats.iterations

        ref, small = render(wavefront_size=1 << 22)
        fill = torch.empty(torch.cuda.mem_get_info()[0] - spare, dtype=torch.uint8, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        for _ in range(2):   # no room for 8 M beside the filling: 4 M, in the workspace at hand
            img, n = render()
            same_film(img, ref)
            assert abs(n - small) <= 2, (n, small)
            assert abs(torch.cuda.mem_get_info()[0] - before) < 64 << 20
        del fill
        torch.cuda.empty_cache()
        img, n = render()
        same_film(img, ref)
        assert n < small - 2, (n, small)   # 8 M: about half the iterations


def test_untuned_large_render_where_its_wavefront_fits_and_where_not():
    import subprocess
    import sys
    from conftest import ROOT
    code = "import sys; sys.path.insert(0, 'tests'); import test_wavefront_edges as t; t.large_render_in_a_full_device()"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_no_bounce_and_no_depth():
    """max_depth 0 renders black, depth 1 only what camera rays see; twice, so
    that the second render replays a kept graph."""
    with Scene(WORLDS["sky"]()) as s:
        assert not s.render(24, 16, 4, 0, kernel=abi.KERNEL_WAVEFRONT).any()
        for _ in range(2):
            same_film(s.render(24, 16, 4, 1, kernel=abi.KERNEL_WAVEFRONT),
                      s.render(24, 16, 4, 1, kernel=abi.KERNEL_MEGAKERNEL))


# --- the opened-up top level --------------------------------------------------------
def mixed_world(n, seed):
    """n entities of changing kind, overlapping: quads, spheres, meshes with a BVH
    and list meshes of up to four triangles."""
    rng = np.random.default_rng(seed)
    w = S.World(name="mixed")
    m = w.add_material("m", S.disney((0.7, 0.7, 0.7), roughness=0.8))
    ico, f = S.icosphere(1)
    for k in range(n):
        c, kind = rng.uniform(-3, 3, 3), (k + seed) % 4
        if kind == 0:
            w.add_quad(c, rng.uniform(-2, 2, 3), rng.uniform(-2, 2, 3), m)
        elif kind == 1:
            w.add_sphere(c, float(rng.uniform(0.4, 1.5)), m)
        else:
            tris = (ico * rng.uniform(0.5, 1.5) + c)[f].reshape(-1, 9)
            w.add_mesh(tris[: 80 if kind == 2 else 1 + seed % 4], m)
    w.lights.append(dict(type=S.LIGHT_DIRECTIONAL, direction=(-1.0, -2.0, -1.0), color=(1, 1, 1), intensity=1.0,
                         shadow_samples=1, angular_radius_deg=0.0))
    w.camera = S.camera((0, 0, -12), (0, 0, 0))
    return w


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 9, 17])
@pytest.mark.parametrize("seed", [0, 1, 2, 3])
def test_walks_over_every_kind_of_top_level(oracle, n, seed):
    """Closest hits (bit for bit) and shadow answers equal the oracle's for lists
    and trees of entities of every kind, on both layouts, also for rays along the
    axes."""
    world = mixed_world(n, seed)
    rays = random_rays(((-4, -4, -4), (4, 4, 4)), 20000, seed=seed)
    axis = rays[:3000].copy()
    axis[:, 3:6] = np.eye(3, dtype=np.float32)[np.arange(3000) % 3] * np.where(np.arange(3000) % 2, 1, -1)[:, None]
    rays = np.ascontiguousarray(np.concatenate([rays, axis]))
    ref = oracle.OracleScene(abi.PackedWorld(world))
    want, _ = ref.trace_closest(rays)
    shadow = rays.copy()
    shadow[:, 6] = 1e-4
    shadow[:, 7] = np.random.default_rng(seed).uniform(0.5, 8.0, rays.shape[0])
    lit = ref.trace_any(shadow)
    with Scene(world) as s:
        for layout in (2, 4):
            hits, out = np.zeros((rays.shape[0], 6), np.int32), np.zeros((rays.shape[0], 3), np.float32)
            abi.check(s.lib.rt_trace_closest(s.h, abi.ptr(rays), rays.shape[0], 1e-4, 3.4028235e38, abi.ptr(hits), layout))
            abi.check(s.lib.rt_trace_any(s.h, abi.ptr(shadow), rays.shape[0], abi.ptr(out), layout))
            hit = want[:, 5] == 1
            assert np.array_equal(hits[:, 5] == 1, hit)
            assert np.array_equal(hits[hit][:, [0, 3, 4]], want[hit][:, [0, 3, 4]])
            assert np.array_equal(out, lit)


def test_sobol_camera_dimensions(oracle):
    """Dimensions 0 and 1 over the whole index range (the superset sum)."""
    rng = np.random.default_rng(1)
    n = 1 << 16
    idx = np.concatenate([np.arange(64), rng.integers(0, 1 << 32, n - 64)]).astype(np.uint32)
    dim = (np.arange(n) & 1).astype(np.uint32)
    seed = rng.integers(0, 1 << 32, n).astype(np.uint32)
    out = np.zeros(n, np.float32)
    abi.check(abi.load().rt_sobol_batch(abi.ptr(idx), abi.ptr(dim), abi.ptr(seed), n, abi.ptr(out)))
    assert np.array_equal(out.view(np.uint32), oracle.sobol(idx, dim, seed).view(np.uint32))


# --- host copies: below a chunk (1 MiB), at its edges, past a window (32 MiB) ----------
@pytest.mark.parametrize("w,h", [(1, 1), (256, 341), (256, 342), (511, 513), (2048, 1366), (2049, 1367)])
def test_display_transform_at_the_copies_edges(w, h):
    """Every pixel arrives and is transformed: against the formula in 64 bits (the
    curve's float steps and powf are a few 2^-24 of a value in [0, 1])."""
    rng = np.random.default_rng(w)
    x = np.exp(rng.normal(-1.0, 1.5, (3, h, w))).astype(np.float32)
    out = np.full((h, w, 3), -1.0, np.float32)
    abi.check(abi.load().rt_tonemap(abi.ptr(x), w, h, 0.5, abi.ptr(out)), "rt_tonemap")
    c = x.astype(np.float64) * float(np.float32(2.0 ** 0.5))
    y = np.clip(c * (2.51 * c + 0.03) / (c * (2.43 * c + 0.59) + 0.14), 0.0, 1.0) ** (1.0 / 2.2)
    np.testing.assert_allclose(out, y.transpose(1, 2, 0), rtol=0, atol=1e-6)


def test_renders_and_display_transforms_from_several_threads():
    """Every caller gets its own film and its own display image, also where the
    staging window and the display buffer are taken by another thread."""
    import threading
    rng = np.random.default_rng(8)
    films = [np.exp(rng.normal(-1.0, 1.5, (3, 400, 700 + k))).astype(np.float32) for k in range(3)]
    lib = abi.load()

    def shown(x):
        out = np.full(x.shape[1:] + (3,), -1.0, np.float32)
        abi.check(lib.rt_tonemap(abi.ptr(x), x.shape[2], x.shape[1], 0.0, abi.ptr(out)), "rt_tonemap")
        return out

    worlds = [WORLDS["cornell"](), WORLDS["icospheres"]()]
    size = dict(w=420, h=300, spp=2, depth=3, kernel=abi.KERNEL_WAVEFRONT)
    alone = [shown(x) for x in films]
    with Scene(worlds[0]) as a, Scene(worlds[1]) as b:
        ref = [s.render(**size) for s in (a, b)]
        wrong = []

        def show(k):
            for _ in range(12):
                if not np.array_equal(shown(films[k]), alone[k]):
                    wrong.append(("display", k))

        def draw(s, want):
            for _ in range(12):
                if not np.allclose(s.render(**size), want, rtol=1e-5, atol=1e-6):
                    wrong.append(("film", s))

        threads = [threading.Thread(target=show, args=(k,)) for k in range(3)]
        threads += [threading.Thread(target=draw, args=(s, r)) for s, r in ((a, ref[0]), (b, ref[1]))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not wrong


def test_kept_memory_is_given_back():
    """After large calls rt_release_memory frees what they left, also from a second
    thread while renders run; films and display images stay what they were."""
    import threading
    import torch
    lib = abi.load()
    x = np.exp(np.random.default_rng(2).normal(-1.0, 1.5, (3, 1080, 1920))).astype(np.float32)
    shown = [np.empty((1080, 1920, 3), np.float32) for _ in range(2)]
    size = dict(w=512, h=384, spp=24, depth=6, kernel=abi.KERNEL_WAVEFRONT)
    with Scene(WORLDS["sky"]()) as s:
        ref = s.render(**size)   # 4.7 M samples: 4 M slots, over 1 GB
        abi.check(lib.rt_tonemap(abi.ptr(x), 1920, 1080, 0.0, abi.ptr(shown[0])), "rt_tonemap")
        before = torch.cuda.mem_get_info()[0]
        abi.check(lib.rt_release_memory(-1), "rt_release_memory")
        assert torch.cuda.mem_get_info()[0] - before > 1 << 30
        assert lib.rt_release_memory(99) == -1 and lib.rt_release_memory(-2) == -1
        same_film(s.render(**size), ref)
        abi.check(lib.rt_tonemap(abi.ptr(x), 1920, 1080, 0.0, abi.ptr(shown[1])), "rt_tonemap")
        assert np.array_equal(*shown)
        stop = threading.Event()

        def release():
            while not stop.is_set():
                abi.check(lib.rt_release_memory(0), "rt_release_memory")

        t = threading.Thread(target=release)
        t.start()
        try:
            for _ in range(10):
                same_film(s.render(**size), ref)
                abi.check(lib.rt_tonemap(abi.ptr(x), 1920, 1080, 0.0, abi.ptr(shown[1])), "rt_tonemap")
                assert np.array_equal(*shown)
        finally:
            stop.set()
            t.join()
