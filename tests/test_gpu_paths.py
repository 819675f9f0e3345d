"""Frames with few rays per bounce level run through the one-launch path
kernel, larger ones and all batches through the wavefront's launches: the
images and ray counts of a render must equal those of a batch of that one
job, for every BVH kind and mode and on both sides of the rule's sizes."""
import numpy as np
import pytest

from helpers import S, bvh_args, random_rays

pytestmark = pytest.mark.gpu

KINDS = ["BVH2", "BVH8_Q8", "BVH4_Q8", "BVH8_F32", "BVH2_Q16", "BVH2_TWO_LEVEL"]
MODES = {
    "lambert": dict(material_mode="MATERIAL_LAMBERT", rng_mode="RNG_PER_SAMPLE", max_bounces=5),
    "stream": dict(material_mode="MATERIAL_REF", rng_mode="RNG_REF_STREAM", max_bounces=9),
    "kahan": dict(material_mode="MATERIAL_REF", rng_mode="RNG_PER_SAMPLE", max_bounces=3, accum_mode="ACCUM_KAHAN"),
    "kahan_stream": dict(material_mode="MATERIAL_REF", rng_mode="RNG_REF_STREAM", max_bounces=4,
                         accum_mode="ACCUM_KAHAN"),
    "one_ray": dict(material_mode="MATERIAL_LAMBERT", rng_mode="RNG_PER_SAMPLE", max_bounces=0),
    "nee": dict(material_mode="MATERIAL_LAMBERT", rng_mode="RNG_PER_SAMPLE", max_bounces=5,
                integrator="INTEGRATOR_PATH_NEE"),
    "nee_stream": dict(material_mode="MATERIAL_LAMBERT", rng_mode="RNG_REF_STREAM", max_bounces=4,
                       integrator="INTEGRATOR_PATH_NEE"),
}


def _both(solrt, ctx, sc, data, w, h, spp, mode, frames=2):
    kw = {k: getattr(solrt, v) if isinstance(v, str) else v for k, v in MODES[mode].items()}
    c = data.camera
    cam = solrt.camera_look_at(c["eye"], c["center"], c["up"], c["vfov"], w / h)
    out = []
    for batch in (False, True):
        img = solrt.Image(ctx, w, h, kw.get("accum_mode", solrt.ACCUM_REF_MIX))
        ctx.reset_stats()
        for f in range(frames):
            p = solrt.render_params(w, h, spp=spp, frame=f, seed=5, miss_mode=solrt.MISS_GRADIENT, **kw)
            if batch:
                b = solrt.Batch(ctx, [(sc, img, cam, p)])
                b.launch()
                ctx.synchronize()
                b.close()
            else:
                solrt.Renderer(ctx).cmd_trace_rays(sc, cam, p, img)
        ctx.synchronize()
        st = ctx.stats()
        assert st.error_flags == 0
        a, r8 = img.read()
        out.append((a.view(np.uint32).copy(), r8.copy(), st.segments, st.paths, st.shadow_segments,
                    st.shadow_unoccluded, st.fp64_fallbacks))
        img.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("kind", KINDS)
def test_render_equals_batch(solrt, ctx, kind, mode):
    for data in (S.cornell(), S.mixed_scene(1, max_tris=1200)[0]):
        sc = solrt.SceneDescription(ctx, data, bvh=getattr(solrt, kind))
        for w, h, spp in ((1, 1, 1), (61, 47, 3)):
            _both(solrt, ctx, sc, data, w, h, spp, mode)
        sc.close()


@pytest.mark.parametrize("mode", ["lambert", "stream", "kahan", "nee"])
def test_render_in_several_passes(solrt, mode):
    """A capacity below the frame's pixels, and one below its samples."""
    data = S.cornell()
    for cap in (1000, 3000, 7000):
        c = solrt.Context(0, path_capacity=cap)
        sc = solrt.SceneDescription(c, data)
        big = solrt.Context(0, path_capacity=1 << 16)
        scb = solrt.SceneDescription(big, data)
        imgs = []
        for cx, s in ((c, sc), (big, scb)):
            kw = {k: getattr(solrt, v) if isinstance(v, str) else v for k, v in MODES[mode].items()}
            cam = solrt.camera_look_at(*(data.camera[k] for k in ("eye", "center", "up", "vfov")), 1.0)
            img = solrt.Image(cx, 50, 50, kw.get("accum_mode", solrt.ACCUM_REF_MIX))
            p = solrt.render_params(50, 50, spp=5, seed=3, **kw)
            solrt.Renderer(cx).cmd_trace_rays(s, cam, p, img)
            cx.synchronize()
            imgs.append(img.read()[0].view(np.uint32).copy())
            img.close()
            s.close()
            cx.close()
        assert np.array_equal(*imgs)


@pytest.mark.parametrize("w,h,spp,mode,tris", [
    (424, 425, 1, "kahan", 0), (425, 425, 1, "kahan", 0),               # 180,200 and 180,625 rays per level
    (479, 478, 1, "kahan", 3000), (479, 479, 1, "kahan", 3000),         # 228,962 and 229,441
    (293, 293, 1, "nee", 3000), (294, 293, 1, "nee", 3000),             # 57,232 and 57,428
    (332, 333, 1, "nee", 0), (333, 333, 1, "nee", 0),                   # 73,704 and 73,926
    (412, 491, 2, "stream", 0),                                         # 80,916 of 202,292 pixels
])
def test_both_sides_of_the_rule(solrt, ctx, w, h, spp, mode, tris):
    data = S.mixed_scene(2, min_tris=tris, max_tris=tris + 1)[0] if tris else S.cornell()
    sc = solrt.SceneDescription(ctx, data)
    _both(solrt, ctx, sc, data, w, h, spp, mode, frames=1)
    sc.close()


def test_moving_scene(solrt, ctx):
    """The larger limit of dynamic scenes: 230,400 rays per level."""
    data = S.soup(2000, seed=3, sigma=0.03)
    sc = solrt.SceneDescription(ctx, data, dynamic=True)
    sc.tlas_regenerate()
    _both(solrt, ctx, sc, data, 480, 480, 1, "kahan", frames=1)
    sc.close()


@pytest.mark.parametrize("tris", [196607, 196608])
@pytest.mark.parametrize("w,h", [(128, 128), (129, 128)])
def test_ao_on_both_sides_of_its_limits(solrt, oracle, ctx, tris, w, h):
    """AO frames change loops from 196,608 triangles on, above 16,384 pixels:
    all equal the oracle."""
    data = S.soup(tris, seed=6, sigma=0.004)
    noise = np.random.default_rng(1).integers(0, 256, (64, 64, 4), dtype=np.uint8)
    ctx.set_blue_noise(noise)
    c = data.camera
    cam = solrt.camera_look_at(c["eye"], c["center"], c["up"], c["vfov"], w / h)
    p = solrt.render_params(w, h, spp=2, max_bounces=3, integrator=solrt.INTEGRATOR_AO)
    sc = solrt.SceneDescription(ctx, data)
    img = solrt.Image(ctx, w, h)
    solrt.Renderer(ctx).cmd_trace_rays(sc, cam, p, img)
    ctx.synchronize()
    want, _, _ = oracle.OracleScene(data).render(cam, p, blue_noise=noise)
    assert np.array_equal(img.read()[0].view(np.uint32), want.view(np.uint32))
    img.close()
    sc.close()


@pytest.mark.parametrize("n", [4096, 4097, 8192, 8193])
@pytest.mark.parametrize("bvh", ["bvh2", "bvh8", "bvh2t"])
def test_rays_on_both_sides_of_the_spread_limit(solrt, oracle, ctx, bvh, n):
    """Up to 8,192 rays (8-wide trees: 4,096) are spread over all warps, from
    there on warps take 32."""
    data = S.soup(600, seed=3, sigma=0.05)
    args = bvh_args(solrt, bvh)
    rays = random_rays(n, -1.0, 1.0, seed=5)
    sc = solrt.SceneDescription(ctx, data, **args)
    got = sc.trace_rays(rays)
    want, _ = oracle.OracleScene(data, two_level=bvh == "bvh2t").trace(rays, brute=True)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    sc.close()


@pytest.mark.parametrize("mode", ["lambert", "nee"])
def test_timing_contexts_time_every_stage(solrt, ctx, mode):
    """A context that times its launches renders small frames stage by stage
    too, so that the stages have their launches and times; same image."""
    data = S.cornell()
    kw = {k: getattr(solrt, v) if isinstance(v, str) else v for k, v in MODES[mode].items()}
    cam = solrt.camera_look_at(*(data.camera[k] for k in ("eye", "center", "up", "vfov")), 1.0)
    p = solrt.render_params(60, 60, spp=2, seed=3, **kw)
    imgs = []
    with solrt.Context(0, path_capacity=1 << 16, enable_timing=True) as timed:
        for c in (timed, ctx):
            sc, img = solrt.SceneDescription(c, data), solrt.Image(c, 60, 60)
            c.reset_stats()
            solrt.Renderer(c).cmd_trace_rays(sc, cam, p, img)
            c.synchronize()
            st = c.stats()
            imgs.append(img.read()[0].view(np.uint32).copy())
            if c is timed:
                shadow = 5 if mode == "nee" else 0
                assert (st.extend_launches, st.shade_launches) == (6 + shadow, 6 + shadow)
                assert min(st.extend_ms, st.shade_ms, st.generate_ms, st.accumulate_ms) > 0.0
            img.close()
            sc.close()
    assert np.array_equal(*imgs)


def _launches(solrt, ctx, sc, data, w, h, bounces):
    """Kernels of one frame: the path kernel and the resolve, or two per bounce
    level, the generate and the resolve."""
    cam = solrt.camera_look_at(*(data.camera[k] for k in ("eye", "center", "up", "vfov")), w / h)
    img = solrt.Image(ctx, w, h)
    p = solrt.render_params(w, h, spp=1, max_bounces=bounces, seed=3, material_mode=solrt.MATERIAL_LAMBERT,
                            rng_mode=solrt.RNG_PER_SAMPLE)
    ctx.reset_stats()
    solrt.Renderer(ctx).cmd_trace_rays(sc, cam, p, img)
    ctx.synchronize()
    n = ctx.stats().launches
    img.close()
    return int(n)


@pytest.mark.parametrize("dynamic", [False, True])
@pytest.mark.parametrize("kind", ["BVH8_Q8", "BVH4_Q8", "BVH8_F32"])
def test_wide_kinds_have_their_limits_when_they_move_too(solrt, ctx, kind, dynamic):
    for data, side in ((S.cornell(), (288, 256)), (S.soup(2000, seed=3, sigma=0.03), (512, 224))):
        sc = solrt.SceneDescription(ctx, data, bvh=getattr(solrt, kind), dynamic=dynamic)
        w, h = side  # 73,728 and 114,688 rays per level
        assert _launches(solrt, ctx, sc, data, w, h, 3) == 2
        assert _launches(solrt, ctx, sc, data, w + 1, h, 3) == 2 + 2 * 4
        _both(solrt, ctx, sc, data, w, h, 1, "kahan", frames=1)
        _both(solrt, ctx, sc, data, w + 1, h, 1, "kahan", frames=1)
        sc.close()


@pytest.mark.parametrize("w", [1024, 1025])
def test_moving_scene_on_both_sides_of_its_limit(solrt, ctx, w):
    """917,504 rays per level: the path kernel up to it, the stages above."""
    data = S.soup(2000, seed=3, sigma=0.03)
    sc = solrt.SceneDescription(ctx, data, dynamic=True)
    sc.tlas_regenerate()
    assert _launches(solrt, ctx, sc, data, w, 896, 3) == (2 if w == 1024 else 10)
    _both(solrt, ctx, sc, data, w, 896, 1, "kahan", frames=1)
    sc.close()


@pytest.mark.parametrize("w", [512, 513])
def test_per_pixel_streams_on_both_sides_of_the_limit(solrt, ctx, w):
    """225,280 and 225,720 pixels over 5 levels: 180,224 and 180,576 rays per level."""
    data = S.cornell()
    sc = solrt.SceneDescription(ctx, data)
    assert _launches(solrt, ctx, sc, data, w, 440, 4) == (2 if w == 512 else 12)
    _both(solrt, ctx, sc, data, w, 440, 2, "kahan_stream", frames=1)
    sc.close()


@pytest.mark.parametrize("mode", ["lambert", "stream", "kahan", "kahan_stream", "nee", "nee_stream"])
def test_stages_in_several_passes(solrt, ctx, mode):
    """The frames of test_render_in_several_passes through the stages (a
    counting context takes no path kernel): pixel chunks, several passes of
    samples, and shadow rays with both."""
    data = S.cornell()
    kw = {k: getattr(solrt, v) if isinstance(v, str) else v for k, v in MODES[mode].items()}
    cam = solrt.camera_look_at(*(data.camera[k] for k in ("eye", "center", "up", "vfov")), 1.0)
    out = []
    for cap in (0, 1000, 3000, 7000):
        with (solrt.Context(0, path_capacity=cap, enable_counters=True) if cap
              else solrt.Context(0, path_capacity=1 << 16)) as c:
            sc = solrt.SceneDescription(c, data)
            img = solrt.Image(c, 50, 50, kw.get("accum_mode", solrt.ACCUM_REF_MIX))
            c.reset_stats()
            for f in range(2):
                p = solrt.render_params(50, 50, spp=5, seed=3, frame=f, **kw)
                solrt.Renderer(c).cmd_trace_rays(sc, cam, p, img)
            c.synchronize()
            st = c.stats()
            if cap:
                assert st.launches > 2 * 2 * (kw["max_bounces"] + 1)
            out.append((img.read()[0].view(np.uint32).copy(), st.segments, st.shadow_segments, st.shadow_unoccluded))
            img.close()
            sc.close()
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0]) and o[1:] == out[0][1:]
