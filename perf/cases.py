"""Performance cases: what programs ask of this path tracer, one dict per case.

`listed()` are fixed cases, `draw(rng)` gives more of the same ranges. A case
names what is done ("do"):

  trace    closest hits of a ray array in device memory (trace_rays_device)
  frame    one rendered frame of a static scene (cmd_trace_rays)
  animate  one frame of a scene whose sections move: set_instances,
           tlas_regenerate, then cmd_trace_rays
  batch    many scenes rendered together (Batch.launch)

`prepare` makes inputs and long-lived objects (context, scene with its BVH,
image, batch) from the seed, `run` is one pass through the public API, and
`exact` recomputes outputs in 64-bit floating point where that is affordable.
Geometry is generated on the GPU and handed over as the host arrays that
SceneDescription takes.
"""
import importlib
import math

import numpy as np
import torch

solrt = importlib.import_module("sol-rs_gb300")
S = solrt.scenes

KINDS = {"bvh2": solrt.BVH2, "bvh8": solrt.BVH8_Q8, "two_level": solrt.BVH2_TWO_LEVEL}
MISS = {"black": solrt.MISS_BLACK, "sky": solrt.MISS_REF_SKY, "gradient": solrt.MISS_GRADIENT}
INTEGRATOR = {"path": solrt.INTEGRATOR_PATH, "nee": solrt.INTEGRATOR_PATH_NEE, "ao": solrt.INTEGRATOR_AO,
              "debug": solrt.INTEGRATOR_DEBUG}


def _frame(name, scene, tris, width, height, spp, bounces, **kw):
    c = dict(name=name, do="frame", scene=scene, tris=tris, width=width, height=height, spp=spp, bounces=bounces,
             kind="bvh2", sah=True, integrator="path", material="lambert", rng="per_sample", accum="mix",
             miss="gradient")
    c.update(kw)
    return c


def listed():
    return [
        # a thousand picking / visibility queries against a small mesh: latency
        dict(name="pick", do="trace", scene="soup", tris=20_000, rays=1_009, kind="bvh2", sah=False),
        # a light-baking sized set of incoherent rays against a million triangles
        dict(name="rays_4m", do="trace", scene="soup", tris=1_000_000, rays=4_194_301, kind="bvh2", sah=True),
        # thumbnail preview of the Cornell box: the smallest frame a UI asks for
        _frame("preview", "cornell", 32, 129, 97, 1, 5, miss="black", sah=False),
        # the interactive example's own frame: 8 samples, 32 bounces, its
        # materials and its one random stream per pixel
        _frame("example_frame", "cornell", 32, 1280, 720, 8, 32, miss="black", sah=False, material="ref",
               rng="ref_stream"),
        # the same settings on a mesh with the sky on
        _frame("mesh_frame", "soup", 150_000, 961, 541, 8, 32, miss="sky", sah=True, material="ref",
               rng="ref_stream"),
        # a final-quality frame of the million-triangle soup (the benchmark's workload)
        _frame("soup_1080p", "soup", 1_000_000, 1920, 1080, 64, 4),
        # a closed scene lit by many small emitters, compensated sums, deep
        # paths, on the compact 8-wide tree
        _frame("tunnel_bvh8", "tunnel", 1_048_576, 1366, 768, 16, 8, miss="sky", accum="kahan", kind="bvh8"),
        # next-event estimation in the same kind of scene
        _frame("tunnel_nee", "tunnel", 262_144, 640, 360, 8, 8, miss="sky", integrator="nee"),
        # the ambient-occlusion example on a mesh: 4 samples, 4 bounces
        _frame("ao", "soup", 300_000, 1280, 720, 4, 4, miss="black", integrator="ao"),
        # moving sections: every frame rebuilds the whole hierarchy
        dict(name="animate_rebuild", do="animate", scene="instances", tris=262_144, sections=64, width=960, height=540,
             spp=2, bounces=4, kind="bvh2", sah=False, mode="rebuild"),
        # moving sections kept as two levels: only the top level is rebuilt
        dict(name="animate_two_level", do="animate", scene="instances", tris=1_048_576, sections=64, width=1280,
             height=720, spp=4, bounces=4, kind="two_level", sah=True, mode="rebuild"),
        # many small jobs of uneven size rendered together
        dict(name="batch", do="batch", scene="mixed", tris=20_000, jobs=24, width=256, height=256, spp=8, bounces=5,
             kind="bvh2", sah=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["trace", "frame", "frame", "frame", "frame", "animate", "batch"])
    if do == "trace":
        return dict(do="trace", scene="soup", tris=_log(rng, 100, 1_000_000), rays=_log(rng, 500, 4_000_000),
                    kind=rng.choice(["bvh2", "bvh2", "bvh8"]), sah=rng.random() < 0.5)
    if do == "animate":
        kind = rng.choice(["bvh2", "bvh2", "two_level"])
        sections = rng.choice([8, 27, 64])
        return dict(do="animate", scene="instances", tris=sections * _log(rng, 100, 16_384), sections=sections,
                    width=_log(rng, 320, 1280), height=_log(rng, 240, 720), spp=_log(rng, 1, 4), bounces=4, kind=kind,
                    sah=kind == "two_level" and rng.random() < 0.5,
                    mode=rng.choice(["rebuild", "rebuild", "refit"]) if kind == "bvh2" else "rebuild")
    if do == "batch":
        return dict(do="batch", scene="mixed", tris=_log(rng, 1_000, 50_000), jobs=rng.randint(2, 24),
                    width=_log(rng, 64, 384), height=_log(rng, 64, 384), spp=_log(rng, 1, 16), bounces=5, kind="bvh2",
                    sah=rng.random() < 0.5)
    integrator = rng.choice(["path", "path", "path", "path", "nee", "ao", "debug"])
    scene = rng.choice(["cornell", "soup", "tunnel"]) if integrator != "nee" else rng.choice(["cornell", "tunnel"])
    tris = 32 if scene == "cornell" else _log(rng, 2_000, 1_000_000)
    stream = integrator == "path" and rng.random() < 0.33
    c = _frame(None, scene, tris, _log(rng, 48, 1920), _log(rng, 48, 1080), _log(rng, 1, 16),
               32 if stream else rng.randint(1, 8), kind=rng.choice(["bvh2", "bvh2", "bvh2", "bvh8"]),
               sah=rng.random() < 0.6, integrator=integrator, miss=rng.choice(["black", "sky", "gradient"]))
    del c["name"]
    if integrator == "path":
        c["material"] = "ref" if stream or rng.random() < 0.3 else "lambert"
        c["rng"] = "ref_stream" if stream else "per_sample"
        c["accum"] = rng.choice(["mix", "mix", "kahan"])
    elif integrator in ("ao", "debug"):
        c["spp"], c["bounces"] = (4, 4) if integrator == "ao" else (1, 1)
    # no dearer than the million-triangle frame: shadow rays and chained
    # samples cost more per segment, and the tube keeps its paths long
    cost = min(c["bounces"] + 1, {"cornell": 4, "soup": 3, "tunnel": 16}[scene])
    cost *= 2.5 if stream or integrator == "nee" else 1.0
    while c["width"] * c["height"] * c["spp"] * cost > 120e6:
        c["spp" if c["spp"] > 1 else "height"] //= 2
    return c


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _vertices(pos, normal, color):
    """ModelVertex records from (n, 3) device tensors."""
    one = torch.ones_like(pos[:, :1])
    v = torch.cat([pos, one, color, one, normal, one, torch.zeros_like(pos), 0 * one], 1)
    return v.float().cpu().numpy().view(S.VERTEX_DTYPE)[:, 0]


def _sections(vertex_counts, index_counts, materials, shared=False):
    secs = np.zeros(len(index_counts), S.SECTION_DTYPE)
    secs["vertex_count"] = vertex_counts
    secs["vertex_offset"] = 0 if shared else np.cumsum(vertex_counts) - vertex_counts
    secs["index_count"] = index_counts
    secs["index_offset"] = np.cumsum(index_counts) - index_counts
    secs["material_index"] = materials
    return secs


def _soup_arrays(n, g, lo=0.0, hi=1.0, sigma=0.005):
    """n small triangles around centroids uniform in [lo, hi]^3, with face
    normals and one albedo each: positions, normals, colours per vertex."""
    cen = lo + (hi - lo) * torch.rand((n, 1, 3), generator=g, device="cuda")
    pos = cen + sigma * torch.randn((n, 3, 3), generator=g, device="cuda")
    nrm = torch.linalg.cross(pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0])
    nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
    alb = 0.2 + 0.6 * torch.rand((n, 1, 3), generator=g, device="cuda")
    return pos.reshape(-1, 3), nrm.repeat_interleave(3, 0), alb.expand(n, 3, 3).reshape(-1, 3)


def _soup(n, seed):
    # the triangle size follows the spacing, as in a mesh of n triangles
    sigma = 0.005 * (1_000_000 / n) ** (1.0 / 3.0)
    v = _vertices(*_soup_arrays(n, _generator(seed), sigma=sigma))
    cam = dict(eye=(0.5, 0.5, -1.2), center=(0.5, 0.5, 0.5), up=(0.0, -1.0, 0.0), vfov=45.0)
    return S.SceneData(v, np.arange(3 * n, dtype=np.uint32), _sections([3 * n], [3 * n], [0]),
                       np.array([S.material(roughness=0.6, metallic=0.3)], S.MATERIAL_DTYPE), None, cam, "soup")


def _tunnel(n, seed):
    """Bumpy tube along +z of about n triangles, 2 % of its quads emissive."""
    n_ang = max(8, int(math.sqrt(n)))
    n_ax = max(1, n // (2 * n_ang))
    g = _generator(seed)
    ang = torch.arange(n_ang, device="cuda") * (2 * math.pi / n_ang)
    z = torch.arange(n_ax + 1, device="cuda") * (200.0 / n_ax)
    phase = 2 * math.pi * torch.rand((6,), generator=g, device="cuda")
    r = torch.ones((n_ax + 1, n_ang), device="cuda")
    for k in range(6):
        r += 0.005 * torch.sin((3 * k + 2) * ang[None] + (1.0 + 1.7 * k) * z[:, None] + phase[k])
    nx, ny = torch.cos(ang)[None].expand_as(r), torch.sin(ang)[None].expand_as(r)
    pos = torch.stack([r * nx, r * ny, z[:, None].expand_as(r)], -1).reshape(-1, 3)
    nrm = torch.stack([-nx, -ny, torch.zeros_like(r)], -1).reshape(-1, 3)
    j, i = torch.meshgrid(torch.arange(n_ax, device="cuda"), torch.arange(n_ang, device="cuda"), indexing="ij")
    i1 = (i + 1) % n_ang
    v00, v01, v10, v11 = j * n_ang + i, j * n_ang + i1, (j + 1) * n_ang + i, (j + 1) * n_ang + i1
    quads = torch.stack([v00, v10, v11, v00, v11, v01], -1).reshape(-1, 6)
    lit = torch.rand((len(quads),), generator=g, device="cuda") < 0.02
    idx = torch.cat([quads[~lit].reshape(-1), quads[lit].reshape(-1)]).cpu().numpy().astype(np.uint32)
    n_lit = 6 * int(lit.sum())
    secs = _sections([len(pos)] * 2, [len(idx) - n_lit, n_lit], [0, 1], shared=True)
    mats = [S.material(base=(0.73,) * 3, roughness=0.8), S.material(emissive=(5.0,) * 3)]
    return S.SceneData(_vertices(pos, nrm, torch.ones_like(pos)), idx, secs, np.array(mats, S.MATERIAL_DTYPE), None,
                       dict(S.TUNNEL_CAMERA), "tunnel")


def _cornell(seed, tris=0):
    """The Cornell box with its two boxes turned, and a soup of `tris` in it."""
    rng = np.random.default_rng(seed)
    d = S.cornell(short_angle=rng.uniform(-30, 30), tall_angle=rng.uniform(-30, 30))
    d.materials["roughness"] = 0.5
    d.materials["metallic"] = 0.2
    if not tris:
        return d
    v = _vertices(*_soup_arrays(tris, _generator(seed), 0.15, 0.85))
    secs = np.concatenate([d.sections, _sections([3 * tris], [3 * tris], [len(d.materials)])])
    secs["vertex_offset"][-1], secs["index_offset"][-1] = len(d.vertices), len(d.indices)
    return S.SceneData(np.concatenate([d.vertices, v]),
                       np.concatenate([d.indices, np.arange(3 * tris, dtype=np.uint32)]), secs,
                       np.concatenate([d.materials, np.array([S.material()], S.MATERIAL_DTYPE)]), None, d.camera,
                       "mixed")


def _instances(n, sections, seed):
    """`sections` soups, each turned in its own cell of a cubic grid, and the
    instances of eight animation frames (a slow turn about y)."""
    side, each = round(sections ** (1.0 / 3.0)), n // sections
    parts = [_soup_arrays(each, _generator(seed * 1000 + k), sigma=0.08 * each ** (-1.0 / 3.0) + 0.005)
             for k in range(sections)]
    v = _vertices(*(torch.cat([p[a] for p in parts]) for a in range(3)))
    idx = np.tile(np.arange(3 * each, dtype=np.uint32), sections)
    secs = _sections([3 * each] * sections, [3 * each] * sections, [0] * sections)
    rng = np.random.default_rng(seed)
    turn = [(rng.normal(size=3), rng.uniform(0, 360)) for _ in range(sections)]
    frames = []
    for f in range(8):
        inst = []
        for k in range(sections):
            cell = np.array([k // (side * side), k // side % side, k % side], np.float64)
            M = np.eye(4)
            M[:3, :3] = S.rotation(*turn[k]) @ S.rotation((0, 1, 0), 5.0 * f) / side
            M[:3, 3] = (cell + 0.5) / side - M[:3, :3] @ np.full(3, 0.5)
            inst.append(S.instance_of(M, k))
        frames.append(np.array(inst, S.INSTANCE_DTYPE))
    cam = dict(eye=(0.5, 0.5, -1.2), center=(0.5, 0.5, 0.5), up=(0.0, -1.0, 0.0), vfov=45.0)
    return S.SceneData(v, idx, secs, np.array([S.material()], S.MATERIAL_DTYPE), frames[0], cam, "instances"), frames


def _scene(case, seed):
    if case["scene"] == "cornell":
        return _cornell(seed)
    return (_soup if case["scene"] == "soup" else _tunnel)(case["tris"], seed)


def _rays(data, n, seed):
    """Rays from uniform points of the scene's box in uniform directions."""
    g = _generator(seed + 1)
    lo, hi = (torch.tensor(f(data.vertices["pos"][:, :3], 0), device="cuda") for f in (np.min, np.max))
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    d = torch.randn((n, 3), generator=g, device="cuda")
    rays[:, 3] = 1e-3
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 1e4
    return rays


def _params(case, seed):
    return solrt.render_params(
        case["width"], case["height"], spp=case["spp"], max_bounces=case["bounces"], seed=seed,
        miss_mode=MISS[case.get("miss", "gradient")],
        material_mode=solrt.MATERIAL_REF if case.get("material") == "ref" else solrt.MATERIAL_LAMBERT,
        rng_mode=solrt.RNG_REF_STREAM if case.get("rng") == "ref_stream" else solrt.RNG_PER_SAMPLE,
        accum_mode=solrt.ACCUM_KAHAN if case.get("accum") == "kahan" else solrt.ACCUM_REF_MIX,
        integrator=INTEGRATOR[case.get("integrator", "path")])


def _camera(data, case):
    c = data.camera
    return solrt.camera_look_at(c["eye"], c["center"], c["up"], c["vfov"], case["width"] / case["height"])


class _DeviceArray:
    """A buffer of an Image, as torch sees it; a tensor made from it holds on
    to the image, whose memory it is."""

    def __init__(self, image, ptr, shape, typestr):
        self.image = image
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _image_tensors(image):
    accum, rgba8 = image.device_ptrs()
    shape = (image.height, image.width, 4)
    return (torch.as_tensor(_DeviceArray(image, accum, shape, "<f4"), device="cuda"),
            torch.as_tensor(_DeviceArray(image, rgba8, shape, "|u1"), device="cuda"))


# ---------------------------------------------------------------------------
# The interface
# ---------------------------------------------------------------------------

def prepare(case, seed):
    seed = seed % 1_000_003
    s = dict(do=case["do"], step=0)
    paths = case.get("width", 0) * case.get("height", 0) * case.get("spp", 1)
    if case["do"] == "batch":
        paths *= case["jobs"]
    # room for a whole frame's paths, as a program sets it up once; at most 2^27
    ctx = s["ctx"] = solrt.Context(0, path_capacity=min(max(paths, 1 << 16), 1 << 27))
    kind, sah = KINDS[case["kind"]], bool(case["sah"])
    if case["do"] == "batch":
        rng = np.random.default_rng(case["jobs"])  # the same sizes whatever the seed
        jobs = []
        for j in range(case["jobs"]):
            scale = math.exp(rng.uniform(-1.0, 1.0))
            data = _cornell(seed * 64 + j, max(64, int(case["tris"] * scale)))
            sc = solrt.SceneDescription(ctx, data, bvh=kind, sah=sah, keep_data=False)
            c = dict(case, width=max(16, int(case["width"] * rng.uniform(0.5, 1.0))),
                     height=max(16, int(case["height"] * rng.uniform(0.5, 1.0))),
                     spp=max(1, int(case["spp"] * rng.uniform(0.5, 1.0))), miss="black")
            jobs.append((sc, solrt.Image(ctx, c["width"], c["height"]), _camera(data, c), _params(c, seed + j)))
        s["batch"] = solrt.Batch(ctx, jobs, graph=True)
        s["out"] = [_image_tensors(job[1]) for job in jobs]
        return s
    if case["do"] == "animate":
        data, s["instances"] = _instances(case["tris"], case["sections"], seed)
    else:
        data = _scene(case, seed)
    s["scene"] = solrt.SceneDescription(ctx, data, bvh=kind, sah=sah, dynamic=case["do"] == "animate",
                                        keep_data=False)
    if case["do"] == "trace":
        s["rays"] = _rays(data, case["rays"], seed)
        s["hits"] = torch.empty((case["rays"], 4), device="cuda")
        return s
    if case.get("integrator") == "ao":
        noise = np.random.default_rng(seed).integers(0, 256, (256, 256, 4), dtype=np.uint8)
        ctx.set_blue_noise(noise)
    s["params"], s["camera"] = _params(case, seed), _camera(data, case)
    s["image"] = solrt.Image(ctx, case["width"], case["height"], s["params"].accum_mode)
    s["renderer"] = solrt.Renderer(ctx)
    s["out"] = _image_tensors(s["image"])
    s["mode"] = solrt.REGEN_REFIT if case.get("mode") == "refit" else solrt.REGEN_REBUILD
    return s


def run(s):
    if s["do"] == "trace":
        s["scene"].trace_rays_device(s["rays"].data_ptr(), len(s["rays"]), s["hits"].data_ptr())
        return dict(t=s["hits"][:, 0], prim=s["hits"].view(torch.int32)[:, 1], u=s["hits"][:, 2], v=s["hits"][:, 3])
    if s["do"] == "batch":
        s["batch"].launch()
        return dict(images=s["out"])
    if s["do"] == "animate":
        s["scene"].set_instances(s["instances"][s["step"] % len(s["instances"])])
        s["scene"].tlas_regenerate(s["mode"])
        # a moving scene starts its accumulation again with every frame
        s["params"].accum_start_frame = s["step"]
    s["params"].frame = s["step"]
    s["renderer"].cmd_trace_rays(s["scene"], s["camera"], s["params"], s["image"])
    s["step"] += 1
    return dict(image=s["out"][0], rgba8=s["out"][1])


def work(case):
    """Bytes: scene, rays and images once. Operations: per ray segment a
    descent of the hierarchy (two boxes of 12 operations per level, and as
    many levels again for the boxes beside the path), two triangle tests and
    the shading."""
    n, jobs = case["tris"], case.get("jobs", 1)
    scene = jobs * n * (36 + 12 + 3 * 36)
    per_segment = 2 * math.ceil(math.log2(n + 1)) * 24 + 2 * 60
    if case["do"] == "trace":
        return dict(bytes=jobs * n * 48 + 48 * case["rays"], flops=case["rays"] * per_segment)
    pixels = jobs * case["width"] * case["height"]
    if case["do"] == "batch":
        pixels = pixels * 0.56
    # mean path length: the box and the tube keep their paths, the soups lose them
    longest = {"cornell": 4.0, "mixed": 4.0, "tunnel": 8.0}.get(case["scene"], 3.0)
    segments = pixels * case["spp"] * min(case["bounces"] + 1.0, longest)
    if case.get("integrator") == "debug":
        segments = pixels
    elif case.get("integrator") == "nee":
        segments *= 2
    flops = segments * (per_segment + 150)
    if case["do"] == "animate":
        scene += 32 * 3 * n  # the moved vertices
        if case["kind"] == "bvh2":  # sort, link and refit every triangle
            scene += n * (48 + 64 + 16)
            flops += 60 * n
    return dict(bytes=scene + pixels * (16 + 4), flops=flops)


# ---------------------------------------------------------------------------
# 64-bit recomputation
# ---------------------------------------------------------------------------

def _closest(tri, org, direc, tmin, tmax):
    """Closest hits by testing every triangle, (t, prim, u, v); a miss keeps
    tmax and prim -1. tri: (n, 3, 3), rays (m, 3), all float64."""
    out_t, out_p, out_u, out_v = [], [], [], []
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    step = max(1, 25_000_000 // len(tri))
    for a in range(0, len(org), step):
        o, d = org[a:a + step, None], direc[a:a + step, None]
        p = torch.linalg.cross(d.expand(-1, len(tri), -1), e2.expand(len(o), -1, -1))
        det = (e1 * p).sum(-1)
        q0 = o - tri[:, 0]
        u = (q0 * p).sum(-1) / det
        q = torch.linalg.cross(q0, e1.expand(len(o), -1, -1))
        v = (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > tmin) & (t < tmax)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        tb, k = t.min(1)
        hit = torch.isfinite(tb)
        zero = torch.zeros_like(tb)
        out_t.append(torch.where(hit, tb, zero + tmax))
        out_p.append(torch.where(hit, k, k * 0 - 1))
        out_u.append(torch.where(hit, u.gather(1, k[:, None])[:, 0], zero))
        out_v.append(torch.where(hit, v.gather(1, k[:, None])[:, 0], zero))
    return torch.cat(out_t), torch.cat(out_p), torch.cat(out_u), torch.cat(out_v)


M32 = 0xFFFFFFFF


def _tea(v0, v1):
    s0 = 0
    for _ in range(16):
        s0 = (s0 + 0x9E3779B9) & M32
        v0 = (v0 + ((((v1 << 4) + 0xA341316C) & M32) ^ ((v1 + s0) & M32) ^ (((v1 >> 5) + 0xC8013EA4) & M32))) & M32
        v1 = (v1 + ((((v0 << 4) + 0xAD90777D) & M32) ^ ((v0 + s0) & M32) ^ (((v0 >> 5) + 0x7E95761E) & M32))) & M32
    return v0


def _mul32(a, b):
    """Low 32 bits of a product of 32-bit values held in int64."""
    return ((a * (b & 0xFFFF)) + (((a * (b >> 16)) & 0xFFFF) << 16)) & M32


def _rand(state):
    state = (_mul32(state, 747796405) + 1) & M32
    word = _mul32((state >> ((state >> 28) + 4)) ^ state, 277803737)
    word = (word >> 22) ^ word
    return state, word.double() / 4294967295.0


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _align(n, cos_t, phi):
    sin_t = (1 - cos_t * cos_t).clamp(0, 1).sqrt()
    x, y, z = n[:, 0], n[:, 1], n[:, 2]
    s = torch.where(z < 0, -1.0, 1.0).double()
    a = -1 / (s + z)
    b = x * y * a
    u = torch.stack([1 + s * x * x * a, s * b, -s * x], -1)
    v = torch.stack([b, s + y * y * a, -y], -1)
    return (u * torch.cos(phi)[:, None] + v * torch.sin(phi)[:, None]) * sin_t[:, None] + n * cos_t[:, None]


def _ggx(n, xi0, xi1, alpha2):
    return _align(n, ((1 - xi0) / (xi0 * (alpha2 - 1) + 1)).clamp(0, 1).sqrt(), 2 * math.pi * xi1)


def _miss(direc, mode):
    one = torch.ones_like(direc[:, :1])
    y = _unit(direc)[:, 1:2]
    rgb = lambda *c: torch.tensor(c, dtype=torch.float64, device=direc.device) * one  # noqa: E731
    if mode == "gradient":
        t = 0.5 * (y + 1)
        return rgb(1, 1, 1) * (1 - t) + rgb(0.5, 0.7, 1.0) * t
    if mode == "sky":
        t = ((0.5 * (y + 1) - 0.35) / 0.3).clamp(0, 1)
        t = t * t * (3 - 2 * t)
        sky = rgb(0.58, 0.45, 0.25) * (1 - t) + rgb(0.3, 0.4, 0.5) * t
        sun = _dot(_unit(direc), _unit(rgb(0.0, 1.0, -0.25))) > 0.99
        return torch.where(sun, rgb(120.0, 100.0, 50.0), sky)
    return 0 * rgb(1, 1, 1)


def _exact_paths(case, seed, data):
    """Mean radiance per pixel of frame 0, path traced in 64 bits with the
    renderer's random streams (sections without transforms)."""
    dev = torch.device("cuda")
    f64 = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    owner = np.repeat(np.arange(len(data.sections)), data.sections["index_count"] // 3)
    vid = data.indices.reshape(-1, 3).astype(np.int64) + data.sections["vertex_offset"][owner].astype(np.int64)[:, None]
    tri, nrm, col = (f64(data.vertices[f][vid][..., :3]) for f in ("pos", "normal", "color"))
    mat = data.materials[data.sections["material_index"][owner]]
    base, emit = f64(mat["base_color"][:, :3]), f64(mat["emissive"])
    metal, rough = f64(mat["metallic"]), f64(mat["roughness"])
    cam, W, H = _camera(data, case), case["width"], case["height"]
    V, P = (f64(m).reshape(4, 4).T for m in (cam.view_inverse, cam.projection_inverse))
    pix = torch.arange(W * H, device=dev)
    tmin = max(1.0, float(V[:3, 3].norm())) * 1e-3
    total = torch.zeros((W * H, 3), dtype=torch.float64, device=dev)
    state = None
    for smp in range(case["spp"]):
        if case["rng"] == "per_sample":
            state = _tea(pix, torch.full_like(pix, smp))
            if seed:
                state = state ^ _tea(torch.tensor(seed, device=dev), torch.tensor(0, device=dev))
        elif smp == 0:
            state = _tea(pix, torch.zeros_like(pix))
        state, jx = _rand(state)
        state, jy = _rand(state)
        ndc = torch.stack([(pix % W + jx) / W * 2 - 1, (pix // W + jy) / H * 2 - 1, 1 + 0 * jx, 1 + 0 * jx], -1)
        direc = _unit((ndc @ P.T)[:, :3]) @ V[:3, :3].T
        org = V[:3, 3].expand(len(pix), 3).contiguous()
        thr = torch.ones_like(org)
        live = pix
        for depth in range(case["bounces"] + 1):
            if not len(live):
                break
            t, prim, u, v = _closest(tri, org, direc, tmin, 1e4)
            k = prim.clamp_min(0)
            miss, light = prim < 0, (prim >= 0) & (emit[k] >= 1).any(1)
            end = torch.where(miss[:, None], _miss(direc, case["miss"]), emit[k]) * thr
            done = miss | light
            total.index_add_(0, live[done], end[done])
            go = ~done
            live, org, direc, thr, k, u, v = (x[go] for x in (live, org, direc, thr, k, u, v))
            b = torch.stack([1 - u - v, u, v], -1)[:, :, None]
            n, hit, c = _unit((nrm[k] * b).sum(1)), (tri[k] * b).sum(1), (col[k] * b).sum(1)
            n = n * torch.sign(-_dot(n, direc))
            s = state[live]
            s, xi0 = _rand(s)
            s, xi1 = _rand(s)
            s, rnd = _rand(s)
            state[live] = s
            new, hue = _align(n, xi0.sqrt(), 2 * math.pi * xi1), base[k] * c
            if case["material"] == "ref":
                alpha2 = rough[k] ** 2
                mirror = lambda d, m: d - 2 * _dot(m, d) * m  # noqa: E731
                mh = _ggx(n, xi0, xi1, alpha2)
                cos_i = _dot(n, mh).abs()[:, 0]
                eta = 1.0 / 1.5
                sin2 = eta * eta * (1 - cos_i * cos_i)
                cos_o = (1 - sin2).clamp(0, 1).sqrt()
                rs, rp = (cos_i - eta * cos_o) / (cos_i + eta * cos_o), (eta * cos_i - cos_o) / (eta * cos_i + cos_o)
                fresnel = torch.where(sin2 <= 1, 0.5 * (rs * rs + rp * rp), torch.ones_like(rs))
                coat = (rnd < fresnel)[:, None]
                new = torch.where(coat, mirror(direc, mh), new)
                hue = torch.where(coat, torch.ones_like(hue), hue)
                shiny = (rnd < metal[k])[:, None]
                new = torch.where(shiny, _ggx(mirror(direc, n), xi0, xi1, alpha2), new)
                hue = torch.where(shiny, base[k] * c, hue)
            thr, org, direc = thr * hue, hit + 1e-4 * n, new
    mean = (total / case["spp"]).reshape(H, W, 3)
    return torch.cat([mean, torch.ones_like(mean[..., :1])], -1)


def exact(case, seed):
    seed = seed % 1_000_003
    if case["do"] == "trace" and case["rays"] * case["tris"] <= 20_000_000_000:
        data = _scene(case, seed)
        rays = _rays(data, case["rays"], seed).double()
        tri = torch.tensor(data.vertices["pos"][:, :3].astype(np.float64).reshape(-1, 3, 3), device="cuda")
        t, prim, u, v = _closest(tri, rays[:, 0:3], rays[:, 4:7], float(np.float32(1e-3)), 1e4)
        return dict(t=t, prim=prim.int(), u=u, v=v)
    if case["do"] == "frame" and case["scene"] == "cornell" and case["integrator"] == "path":
        if case["width"] * case["height"] * case["spp"] <= 20_000_000:
            return dict(image=_exact_paths(case, seed, _cornell(seed)), rgba8=None)
    return None
