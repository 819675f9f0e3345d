"""BVH2 scenes traverse a 32-byte copy of their nodes when it pays (from 512
triangles on, unless the scene's 16-bit grid is too coarse for them): hit
records stay those of the oracle's brute force on both sides of each rule,
through builds, refits and batches that mix both."""
import numpy as np
import pytest

from helpers import S

pytestmark = pytest.mark.gpu


def _rays(rng, data, n):
    pos = data.vertices["pos"][data.indices][:, :3].astype(np.float64)
    tri = pos.reshape(-1, 3, 3)
    k = rng.integers(0, len(tri), n)
    b = rng.dirichlet((1, 1, 1), n)
    target = (tri[k] * b[:, :, None]).sum(1)   # points on triangles, some on edges
    target[: n // 8] = tri[k[: n // 8], 0]      # and some on vertices
    d = rng.normal(size=(n, 3))
    d[n // 2:: 16, 0] = 0.0                     # axis-parallel components
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ext = np.linalg.norm(tri.max((0, 1)) - tri.min((0, 1)))
    rays = np.zeros(n, [("origin", "<f4", 3), ("tmin", "<f4"), ("dir", "<f4", 3), ("tmax", "<f4")])
    rays["origin"] = target - d * (rng.random((n, 1)) * 0.3 * ext)
    rays["dir"] = d
    rays["tmin"], rays["tmax"] = 1e-5 * ext, 1e4 * ext
    return rays


def _stretched(n, far):
    """A soup of n triangles and two that stretch the scene's box to +-far."""
    d = S.soup(n, seed=11, sigma=0.05)
    v = d.vertices.copy()
    v["pos"][0:3, :3] = [[far, far, far], [far + 0.1, far, far], [far, far + 0.1, far]]
    v["pos"][3:6, :3] = [[-far, -far, -far], [0.1 - far, -far, -far], [-far, 0.1 - far, -far]]
    return S.SceneData(v, d.indices, d.sections, d.materials, None, d.camera, "stretched")


def _moved(n, offset, scale):
    d = S.soup(n, seed=12, sigma=0.05)
    v = d.vertices.copy()
    v["pos"][:, :3] = v["pos"][:, :3] * np.float32(scale) + np.float32(offset)
    return S.SceneData(v, d.indices, d.sections, d.materials, None, d.camera, "moved")


@pytest.mark.parametrize("maker", [
    lambda: S.soup(511, seed=1, sigma=0.05), lambda: S.soup(512, seed=1, sigma=0.05),
    lambda: S.soup(513, seed=1, sigma=0.05), lambda: S.soup(3001, seed=2, sigma=0.03),
    lambda: _stretched(2000, 3.0), lambda: _stretched(2000, 1e3), lambda: _stretched(2000, 1e7),
    lambda: _moved(2000, 1000.0, 1.0), lambda: _moved(2000, 0.0, 1e-6), lambda: _moved(2000, -3e5, 1e4),
    lambda: S.tunnel(n_ang=64, n_ax=32, length=300.0),
], ids=["511", "512", "513", "3001", "far3", "far1e3", "far1e7", "off1000", "tiny", "off3e5", "tunnel"])
@pytest.mark.parametrize("sah", [False, True])
def test_hits_equal_brute_force(solrt, oracle, ctx, maker, sah):
    d = maker()
    rays = _rays(np.random.default_rng(5), d, 4096).view(solrt.RAY_DTYPE)
    sc = solrt.SceneDescription(ctx, d, sah=sah)
    got = sc.trace_rays(rays)
    want, _ = oracle.OracleScene(d).trace(rays, brute=True)
    for f in ("prim", "t", "u", "v"):
        assert np.array_equal(got[f].view(np.uint32), want[f].view(np.uint32)), f
    sc.close()


def test_non_finite_vertices_do_not_hide_the_rest(solrt, oracle, ctx):
    """A vertex at infinity leaves no finite grid: the scene still gives the
    oracle's hits."""
    d = S.soup(1000, seed=3, sigma=0.05)
    v = d.vertices.copy()
    v["pos"][7, 1] = np.inf
    d = S.SceneData(v, d.indices, d.sections, d.materials, None, d.camera, "inf")
    rays = _rays(np.random.default_rng(6), S.soup(1000, seed=3, sigma=0.05), 2048).view(solrt.RAY_DTYPE)
    sc = solrt.SceneDescription(ctx, d)
    got = sc.trace_rays(rays)
    want, _ = oracle.OracleScene(d).trace(rays, brute=True)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    sc.close()


def test_batch_mixing_both_node_formats(solrt, ctx):
    """One batch over a scene below and one above the size rule, then updated
    with cameras swapped: each image equals its own render."""
    scenes = [solrt.SceneDescription(ctx, d) for d in (S.cornell(), S.soup(4000, seed=4, sigma=0.03))]
    cams = [solrt.camera_look_at(sc.data.camera["eye"], sc.data.camera["center"], sc.data.camera["up"],
                                 sc.data.camera["vfov"], 1.0) for sc in scenes]
    p = solrt.render_params(40, 40, spp=3, max_bounces=4, seed=9, miss_mode=solrt.MISS_GRADIENT,
                            material_mode=solrt.MATERIAL_LAMBERT, rng_mode=solrt.RNG_PER_SAMPLE)
    for pick in ((0, 1), (1, 1)):
        jobs = [(scenes[k], solrt.Image(ctx, 40, 40), cams[k], p) for k in pick]
        b = solrt.Batch(ctx, jobs, graph=True)
        for _ in range(2):
            b.launch()
            ctx.synchronize()
            for sc, img, cam, q in jobs:
                alone = solrt.Image(ctx, 40, 40)
                solrt.Renderer(ctx).cmd_trace_rays(sc, cam, q, alone)
                ctx.synchronize()
                assert np.array_equal(img.read()[0].view(np.uint32), alone.read()[0].view(np.uint32))
                alone.close()
            b.update(jobs)
        b.close()


@pytest.mark.parametrize("scale,length", [(1.0, 1e-12), (1.0, 1e-18), (1.0, 1e-20), (1.0, 1e-21), (1.0, 1e-22),
                                          (1.0, 1e-23), (1e6, 1e-20), (1.0, 1e14), (1.0, 1e25), (1.0, 1e33)])
@pytest.mark.parametrize("kind", ["BVH2", "BVH2_Q16"])
def test_short_and_long_axis_parallel_directions(solrt, oracle, ctx, kind, scale, length):
    """A direction component of zero is traced as a tiny one; next to a short
    direction that must not tilt the ray out of the boxes on its way. 1e6: a
    scene whose grid has cells above 8."""
    rng = np.random.default_rng(8)
    d = _moved(2000, 0.0, scale)
    tri = d.vertices["pos"][d.indices][:, :3].astype(np.float64).reshape(-1, 3, 3)
    n = 1200
    k = rng.integers(0, len(tri), n)
    target = (tri[k] * rng.dirichlet((1, 1, 1), n)[:, :, None]).sum(1)
    dirs = np.zeros((n, 3))
    axis = rng.integers(0, 3, n)
    dirs[np.arange(n), axis] = rng.choice([-1.0, 1.0], n)          # along an axis
    dirs[n // 2:, :] += np.roll(dirs[n // 2:, :], 1, axis=1) * 0.7  # in a coordinate plane
    rays = np.zeros(n, solrt.RAY_DTYPE)
    rays["origin"] = target - dirs * rng.uniform(0.1, 1.5, (n, 1)) * scale
    rays["dir"] = dirs * length
    rays["tmax"] = 1e30
    sc = solrt.SceneDescription(ctx, d, bvh=getattr(solrt, kind))
    got = sc.trace_rays(rays)
    want, _ = oracle.OracleScene(d).trace(rays, brute=True)
    assert (want["prim"] != solrt.NO_HIT).mean() > 0.9
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    sc.close()


def _sections(counts):
    """One soup section of each count, all with the identity instance."""
    b = S._Builder()
    for k, n in enumerate(counts):
        S.soup(n, seed=20 + k, sigma=0.05, builder=b)
    data = b.build(S.soup(1).camera, "sections")
    data.instances = np.array([S.instance_of(np.eye(4), k) for k in range(len(counts))], S.INSTANCE_DTYPE)
    return data


def _moved_section(data, k, x):
    """data's instances with section k moved by x along x."""
    inst = data.instances.copy()
    M = np.eye(4)
    M[0, 3] = x
    inst[k] = S.instance_of(M, k)
    return inst


@pytest.mark.parametrize("far", [1e13, 1e30, 3e38])
@pytest.mark.parametrize("mode", ["REGEN_REBUILD", "REGEN_REFIT"])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_launched_again_after_a_section_left_the_grid(solrt, ctx, graph, mode, far):
    """A batch goes on with the nodes it was planned with: the sections that
    stayed are still there when another one has moved beyond every 16-bit
    grid."""
    data = _sections((700, 50))
    sc = solrt.SceneDescription(ctx, data, dynamic=True)
    c = data.camera
    cam = solrt.camera_look_at(c["eye"], c["center"], c["up"], c["vfov"], 1.0)
    p = solrt.render_params(48, 48, spp=2, max_bounces=4, seed=9, miss_mode=solrt.MISS_GRADIENT,
                            material_mode=solrt.MATERIAL_LAMBERT, rng_mode=solrt.RNG_PER_SAMPLE)
    imgs = [solrt.Image(ctx, 48, 48) for _ in range(2)]
    b = solrt.Batch(ctx, [(sc, imgs[0], cam, p)], graph=graph)
    for inst in (data.instances, _moved_section(data, 1, far)):
        sc.set_instances(inst)
        sc.tlas_regenerate(getattr(solrt, mode))
        for img in imgs:
            img.clear()
        b.launch()
        solrt.Renderer(ctx).cmd_trace_rays(sc, cam, p, imgs[1])
        ctx.synchronize()
        got, want = (img.read()[0].view(np.uint32) for img in imgs)
        assert np.array_equal(got, want)
    b.close()
    sc.close()


def _kind(ctx):
    """Nodes that the context's last traversal launch read."""
    out = np.zeros(1, np.uint32)
    ctx.debug_unit(10, 1, out_u=out)
    return int(out[0])


def _with_infinity():
    d = S.soup(1000, seed=3, sigma=0.05)
    v = d.vertices.copy()
    v["pos"][7, 1] = np.inf
    return S.SceneData(v, d.indices, d.sections, d.materials, None, d.camera, "inf")


@pytest.mark.parametrize("maker,copy", [
    (lambda: S.soup(511, seed=1, sigma=0.05), False), (lambda: S.soup(512, seed=1, sigma=0.05), True),
    (lambda: S.soup(3001, seed=2, sigma=0.03), True), (lambda: _stretched(2000, 3.0), True),
    (lambda: _stretched(2000, 1e3), False), (lambda: _stretched(2000, 1e7), False),
    (lambda: _moved(2000, 0.0, 1e-6), True), (lambda: _moved(2000, 0.0, 3e5), True),
    (lambda: _moved(2000, 0.0, 1e6), False), (lambda: _moved(2000, 9e6, 1e4), False), (_with_infinity, False),
    (lambda: S.tunnel(n_ang=64, n_ax=32, length=300.0), True),
], ids=["511", "512", "3001", "far3", "far1e3", "far1e7", "tiny", "cells8", "cells32", "off9e6", "inf", "tunnel"])
def test_which_scenes_traverse_the_copy(solrt, ctx, maker, copy):
    """Rays and frames read the copy where the rules take it; debug frames keep
    the 64-byte nodes."""
    d = maker()
    sc = solrt.SceneDescription(ctx, d)
    want = solrt.BVH2_Q16 if copy else solrt.BVH2
    sc.trace_rays(np.zeros(1, solrt.RAY_DTYPE))
    assert _kind(ctx) == want
    cam = solrt.camera_look_at((0.5, 0.5, -1.2), (0.5, 0.5, 0.5), (0.0, -1.0, 0.0), 45.0, 1.0)
    img = solrt.Image(ctx, 16, 16)
    for integrator, kind in ((solrt.INTEGRATOR_DEBUG, solrt.BVH2), (solrt.INTEGRATOR_PATH, want)):
        solrt.Renderer(ctx).cmd_trace_rays(sc, cam, solrt.render_params(16, 16, spp=1, integrator=integrator), img)
        assert _kind(ctx) == kind
    img.close()
    sc.close()


@pytest.mark.parametrize("mode", ["REGEN_REBUILD", "REGEN_REFIT"])
@pytest.mark.parametrize("how", [{}, dict(graph=True), dict(cooperative=True), dict(cooperative=True, graph=True)],
                         ids=["launches", "graph", "coop", "coop_graph"])
def test_batch_follows_a_scene_over_the_growth_limit(solrt, ctx, how, mode):
    """A section moves away until the grid is too coarse for the others, and
    back: the updated batch (its graph captured again) changes nodes each time
    and renders what a lone frame does."""
    data = _sections((700, 50))
    sc = solrt.SceneDescription(ctx, data, dynamic=True)
    small = solrt.SceneDescription(ctx, S.soup(600, seed=30, sigma=0.05))
    c = data.camera
    cam = solrt.camera_look_at(c["eye"], c["center"], c["up"], c["vfov"], 1.0)
    p = solrt.render_params(48, 48, spp=2, max_bounces=4, seed=9, miss_mode=solrt.MISS_GRADIENT,
                            material_mode=solrt.MATERIAL_LAMBERT, rng_mode=solrt.RNG_PER_SAMPLE)
    jobs = [(s, solrt.Image(ctx, 48, 48), cam, p) for s in (sc, small)]
    alone = solrt.Image(ctx, 48, 48)
    b = solrt.Batch(ctx, jobs, **how)
    b.launch()
    for x, kind in ((3000.0, solrt.BVH2), (0.0, solrt.BVH2_Q16), (3000.0, solrt.BVH2), (1.0, solrt.BVH2_Q16)):
        sc.set_instances(_moved_section(data, 1, x))
        sc.tlas_regenerate(getattr(solrt, mode))
        b.update(jobs)
        for turn in range(2):
            for job in jobs:
                job[1].clear()
            b.launch()
            if not how.get("graph") or turn == 0:
                assert _kind(ctx) == kind
        for s, img, _, _ in jobs:
            alone.clear()
            solrt.Renderer(ctx).cmd_trace_rays(s, cam, p, alone)
            ctx.synchronize()
            assert _kind(ctx) == (kind if s is sc else solrt.BVH2_Q16)
            assert np.array_equal(img.read()[0].view(np.uint32), alone.read()[0].view(np.uint32))
    b.close()
    small.close()
    sc.close()
