"""Calls that fail on the host in the middle of a render or a build (the
failure is made there, solrt_debug_unit op 9) leave the context usable: what
comes after is what a fresh context gives."""
import numpy as np
import pytest

from helpers import S, camera_of

pytestmark = pytest.mark.gpu

ALLOC, LAUNCH = 0, 1


def _let_fail(ctx, site, nth):
    """The nth call of the site from now on fails; what was left of the last count."""
    left = np.zeros(1, np.uint32)
    ctx.debug_unit(9, 1, a=np.array([site], np.uint32), b=np.array([nth], np.uint32), out_u=left)
    return int(left[0])


@pytest.fixture
def wavefront(solrt):
    c = solrt.Context(0, path_capacity=1 << 20, enable_counters=True)  # counting contexts render stage by stage
    yield c
    _let_fail(c, LAUNCH, 0)
    c.close()


@pytest.mark.parametrize("integrator", ["INTEGRATOR_PATH", "INTEGRATOR_PATH_NEE"])
@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_pass_that_ends_early_leaves_no_paths_behind(solrt, ctx, wavefront, nth, integrator):
    data = S.cornell()
    cam = camera_of(data, 1.0)
    p = solrt.render_params(60, 60, spp=3, max_bounces=4, seed=5, material_mode=solrt.MATERIAL_LAMBERT,
                            rng_mode=solrt.RNG_PER_SAMPLE, integrator=getattr(solrt, integrator))
    out = []
    for c, fail in ((wavefront, True), (ctx, False)):
        sc, img = solrt.SceneDescription(c, data), solrt.Image(c, 60, 60)
        if fail:
            _let_fail(c, LAUNCH, nth)
            with pytest.raises(solrt.SolrtError):
                solrt.Renderer(c).cmd_trace_rays(sc, cam, p, img)
            assert _let_fail(c, LAUNCH, 0) == 0
            c.synchronize()
            img.clear()
        c.reset_stats()
        solrt.Renderer(c).cmd_trace_rays(sc, cam, p, img)
        c.synchronize()
        st = c.stats()
        assert st.error_flags == 0
        out.append((img.read()[0].view(np.uint32).copy(), st.segments, st.shadow_segments))
        img.close()
        sc.close()
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]


@pytest.mark.parametrize("graph", [False, True])
def test_batch_after_a_failed_launch(solrt, ctx, graph):
    data = S.cornell()
    cam = camera_of(data, 1.0)
    p = solrt.render_params(40, 40, spp=2, max_bounces=4, seed=5, material_mode=solrt.MATERIAL_LAMBERT,
                            rng_mode=solrt.RNG_PER_SAMPLE)
    sc = solrt.SceneDescription(ctx, data)
    img, alone = solrt.Image(ctx, 40, 40), solrt.Image(ctx, 40, 40)
    b = solrt.Batch(ctx, [(sc, img, cam, p)], graph=graph)
    _let_fail(ctx, LAUNCH, 3)
    with pytest.raises(solrt.SolrtError):
        b.launch()
    assert _let_fail(ctx, LAUNCH, 0) == 0
    ctx.synchronize()
    img.clear()
    b.launch()
    solrt.Renderer(ctx).cmd_trace_rays(sc, cam, p, alone)
    ctx.synchronize()
    assert np.array_equal(img.read()[0].view(np.uint32), alone.read()[0].view(np.uint32))
    b.close()
    sc.close()


def _rays(data, n=2000):
    rng = np.random.default_rng(4)
    rays = np.zeros(n, [("origin", "<f4", 3), ("tmin", "<f4"), ("dir", "<f4", 3), ("tmax", "<f4")])
    rays["origin"] = rng.uniform(-0.2, 1.2, (n, 3))
    d = rng.normal(size=(n, 3))
    rays["dir"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["tmax"] = 1e4
    return rays


def test_every_allocation_of_a_build_may_fail(solrt, oracle):
    """Without memory for the 32-byte copy of its nodes a BVH2 scene keeps the
    64-byte ones; any other missing array is SOLRT_ERR_OOM, and the next
    creation works."""
    data = S.soup(1500, seed=3, sigma=0.05)
    rays = _rays(data)
    want, _ = oracle.OracleScene(data).trace(rays.view(solrt.RAY_DTYPE), brute=True)
    sizes = {}
    for nth in range(1, 100):
        c = solrt.Context(0, path_capacity=1 << 16)
        _let_fail(c, ALLOC, nth)
        try:
            sc = solrt.SceneDescription(c, data)
        except solrt.SolrtError as e:
            assert e.status == 2
            assert _let_fail(c, ALLOC, 0) == 0
            sc = solrt.SceneDescription(c, data)
        else:
            left = _let_fail(c, ALLOC, 0)
            sizes[nth] = (left, sc.device_bytes())
        assert np.array_equal(sc.trace_rays(rays.view(solrt.RAY_DTYPE)).view(np.uint32), want.view(np.uint32))
        sc.close()
        c.close()
        if sizes.get(nth, (0, 0))[0]:
            break
    *without, last = sorted(sizes)  # last: no allocation failed
    assert len(without) == 1 and sizes[without[0]] == (0, sizes[last][1] - 32 * 1500)


def _without_copy(solrt, data):
    """A context and a moving scene on it that had no memory for the copy."""
    for nth in range(1, 100):
        c = solrt.Context(0, path_capacity=1 << 16)
        _let_fail(c, ALLOC, nth)
        try:
            sc = solrt.SceneDescription(c, data, dynamic=True)
        except solrt.SolrtError:
            sc = None
        assert _let_fail(c, ALLOC, 0) == 0
        if sc:
            return c, sc
        c.close()


def _two_sections():
    b = S._Builder()
    for k in range(2):
        S.soup(600, seed=7 + k, sigma=0.05, builder=b)
    data = b.build(S.soup(1).camera, "two")
    data.instances = np.array([S.instance_of(np.eye(4), k) for k in range(2)], S.INSTANCE_DTYPE)
    return data


def test_moving_scene_without_memory_for_the_copy(solrt, ctx):
    """Refits and rebuilds of a scene that was created without the copy take it
    once there is memory, and render the same either way."""
    data = _two_sections()
    plain = solrt.SceneDescription(ctx, data, dynamic=True)
    full = plain.device_bytes()
    cam = camera_of(data, 1.0)
    p = solrt.render_params(40, 40, spp=2, max_bounces=3, seed=5, material_mode=solrt.MATERIAL_LAMBERT,
                            rng_mode=solrt.RNG_PER_SAMPLE)
    c, sc = _without_copy(solrt, data)
    assert sc.device_bytes() == full - 32 * 1200
    want = solrt.Image(ctx, 40, 40)
    solrt.Renderer(ctx).cmd_trace_rays(plain, cam, p, want)
    img = solrt.Image(c, 40, 40)
    for mode, refuse in ((solrt.REGEN_REFIT, True), (solrt.REGEN_REBUILD, False), (solrt.REGEN_REFIT, False)):
        sc.set_instances(data.instances)
        _let_fail(c, ALLOC, 1 if refuse else 0)
        sc.tlas_regenerate(mode)
        _let_fail(c, ALLOC, 0)
        img.clear()
        solrt.Renderer(c).cmd_trace_rays(sc, cam, p, img)
        c.synchronize()
        ctx.synchronize()
        assert np.array_equal(img.read()[0].view(np.uint32), want.read()[0].view(np.uint32))
    assert sc.device_bytes() == full
    sc.close()
    c.close()
    plain.close()


def test_server_frees_what_a_scene_counted_with(solrt):
    """A served scene that grows by its copy between two jobs leaves no bytes
    in use, and none below zero."""
    data = _two_sections()
    c, sc = _without_copy(solrt, data)
    cam = camera_of(data, 1.0)
    p = solrt.render_params(32, 32, spp=1, max_bounces=2, material_mode=solrt.MATERIAL_LAMBERT,
                            rng_mode=solrt.RNG_PER_SAMPLE)
    srv = solrt.Server(c)
    small = sc.device_bytes()
    t = srv.submit(sc, cam, p)
    assert srv.wait(t, 60000).status == 0
    sc.tlas_regenerate(solrt.REGEN_REFIT)
    assert sc.device_bytes() > small
    srv.release(t)
    assert srv.stats().bytes_in_use == 0
    srv.close()
    sc.close()
    c.close()
