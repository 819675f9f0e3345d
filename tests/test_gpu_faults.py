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
