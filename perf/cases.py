"""The renderer's work as its users call it, for timing.

Each case is one call of the public interface on a scene that the caller
already holds: the integrators' ``Render`` (path tracing, volumetric path
tracing, light tracing), batched renders, the differentiable renderer's
forward and backward pass, and ray queries. Contexts are kept per pool size
and BVH width, as a program keeps them; scenes are built anew for every seed
(albedos, roughness, radiance, surface displacement, camera and sphere
positions change with it, sizes do not).
"""
import dataclasses
import math

import numpy as np
import torch

import gyunity_b200 as g
from gyunity_b200 import diff, scenes

_CONTEXTS = {}
_SPHERES = {}
_SKIES = {}

DEFAULT_POOL = 1 << 21   # the library's default number of paths in flight
LARGE_POOL = 1 << 24     # what the single-scene benchmarks use


def listed():
    return [
        # the smallest render, a thumbnail or a preview while a camera moves: launches and latency
        dict(name="thumbnail", kind="path", scene="cornell", res_x=64, res_y=64, spp=4, depth=8, rr=3,
             sampler="sobol", width=2, pool=DEFAULT_POOL),
        # the reference's own Cornell box at its usual size, on a default context
        dict(name="cornell", kind="path", scene="cornell", res_x=256, res_y=256, spp=16, depth=8, rr=3,
             sampler="sobol", width=2, pool=DEFAULT_POOL),
        # every lobe kind, the other sampler, a ragged film and sample count
        dict(name="mixed_halton", kind="path", scene="mixed", res_x=333, res_y=217, spp=7, depth=8, rr=3,
             sampler="halton", width=2, pool=DEFAULT_POOL, level=4),
        # a large mesh of glossy metal, final quality: the single-scene benchmark's scene at fewer samples
        dict(name="mesh", kind="path", scene="mesh", res_x=1024, res_y=1024, spp=16, depth=16, rr=5,
             sampler="sobol", width=8, pool=LARGE_POOL, level=8),
        # a full HD frame of rough glass under a sky map: many camera rays miss
        dict(name="sky_glass", kind="path", scene="knot", res_x=1920, res_y=1080, spp=16, depth=32, rr=5,
             sampler="sobol", width=8, pool=LARGE_POOL, level=250, env=2048),
        # many uneven scenes in one call, the headline workload at fewer instances
        dict(name="batch", kind="batch", instances=16, salt=1, max_res=1024, max_spp=64, max_level=7, depth=16, rr=5,
             sampler="sobol", width=8, pool=LARGE_POOL),
        # the same call for a sheet of small previews
        dict(name="batch_previews", kind="batch", instances=24, salt=2, max_res=96, max_spp=4, max_level=4, depth=8,
             rr=5, sampler="sobol", width=2, pool=DEFAULT_POOL),
        # a room in fog, the volumetric integrator's default (equi-angular) estimator
        dict(name="fog", kind="volume", scene="fog", res_x=512, res_y=512, spp=8, depth=8, equi=True,
             sampler="sobol", width=2, pool=DEFAULT_POOL),
        # a ball of fog entered through its faces, distance sampling, ragged film
        dict(name="fog_ball", kind="volume", scene="fog_ball", res_x=203, res_y=151, spp=6, depth=6, equi=False,
             sampler="sobol", width=2, pool=DEFAULT_POOL, level=2),
        # light tracing: splats all over the film
        dict(name="light_tracing", kind="light", scene="cornell", res_x=512, res_y=512, spp=16, depth=8,
             sampler="sobol", width=2, pool=DEFAULT_POOL),
        # one inverse-rendering step: image, loss, gradients of 1036 parameters
        dict(name="inverse_step", kind="adjoint", res_x=256, res_y=256, spp=16, depth=8, level=5, groups=256,
             sampler="sobol", width=2, pool=DEFAULT_POOL),
        # a host program's own ray queries (picking, visibility), closest hit
        dict(name="ray_queries", kind="rays", scene="mesh", rays=262147, width=2, pool=DEFAULT_POOL, level=5,
             any_hit=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges, at most 16M paths."""
    kind = rng.choice(["path", "path", "path", "path", "batch", "volume", "light", "adjoint", "rays"])
    width = rng.choice([2, 8])
    pool = rng.choice([DEFAULT_POOL, DEFAULT_POOL, 1 << 22, LARGE_POOL])
    sampler = rng.choice(["sobol", "sobol", "halton"])
    res_x, res_y = _log_int(rng, 40, 1400), _log_int(rng, 40, 1100)
    spp = _log_int(rng, 1, 64)
    spp = max(1, min(spp, (1 << 24) // (res_x * res_y)))
    base = dict(kind=kind, width=width, pool=pool, sampler=sampler)
    if kind == "path":
        scene = rng.choice(["cornell", "mixed", "mesh", "knot"])
        c = dict(base, scene=scene, res_x=res_x, res_y=res_y, spp=spp, depth=rng.randint(2, 24), rr=rng.randint(2, 6))
        if scene == "mixed":
            c["level"] = rng.randint(2, 6)
        elif scene == "mesh":
            c["level"] = rng.randint(2, 8)
        elif scene == "knot":
            c.update(level=_log_int(rng, 12, 250), env=rng.choice([128, 512, 1500, 2048]))
        return c
    if kind == "batch":
        return dict(base, instances=rng.randint(1, 30), salt=rng.randint(3, 1 << 20), max_res=_log_int(rng, 64, 400),
                    max_spp=_log_int(rng, 1, 16), max_level=rng.randint(3, 7), depth=rng.randint(4, 16), rr=5)
    if kind == "volume":
        return dict(base, scene=rng.choice(["fog", "fog_ball"]), res_x=min(res_x, 700), res_y=min(res_y, 600),
                    spp=min(spp, 12), depth=rng.randint(2, 10), equi=rng.choice([True, False]), level=rng.randint(1, 4))
    if kind == "light":
        return dict(base, scene=rng.choice(["cornell", "mixed"]), res_x=min(res_x, 700), res_y=min(res_y, 600),
                    spp=min(spp, 24), depth=rng.randint(2, 10), level=rng.randint(2, 5))
    if kind == "adjoint":
        return dict(base, res_x=min(res_x, 400), res_y=min(res_y, 400), spp=min(spp, 16), depth=rng.randint(2, 8),
                    level=rng.randint(3, 5), groups=rng.choice([1, 7, 64, 256]))
    return dict(base, scene=rng.choice(["mesh", "cornell"]), rays=_log_int(rng, 1, 1_000_000),
                level=rng.randint(2, 7), any_hit=rng.choice([False, False, True]))


# ------------------------------------------------------------------ scenes ---
def _context(case):
    key = (case["pool"], case["width"])
    if key not in _CONTEXTS:
        _CONTEXTS[key] = g.Context(0, capacity=case["pool"], bvh_width=case["width"])
    return _CONTEXTS[key]


def _unit_sphere(level):
    if level not in _SPHERES:
        _SPHERES[level] = scenes.icosphere(level)
    return _SPHERES[level]


def _ripple(points, rng, terms=6):
    """A smooth seeded displacement in about [-1, 1]."""
    out = np.zeros(points.shape[0])
    for k in range(terms):
        d = rng.normal(size=3) * (2.0 + 2.0 * k)
        out += np.sin(points @ d + rng.uniform(0, 2 * np.pi)) / terms
    return out


def _smooth_normals(v, f):
    fn = np.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])
    idx = f.reshape(-1)
    n = np.stack([np.bincount(idx, np.repeat(fn[:, a], 3), minlength=v.shape[0]) for a in range(3)], 1)
    return (n / np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-30)).astype(np.float32)


def _ball(level, radius, center, rng):
    v, f = _unit_sphere(level)
    p = (v * (radius * (1.0 + 0.05 * _ripple(v, rng)))[:, None] + np.asarray(center)).astype(np.float32)
    return p, _smooth_normals(p.astype(np.float64), f), f


def _material(kind, a=(0, 0, 0), b=(0, 0, 0), alpha=0.0):
    p = np.zeros(16, np.float32)
    p[0:3], p[3:6], p[6], p[7], p[8], p[9:12], p[12:15], p[15] = a, b, alpha, alpha, 1.5, 1.5, 1.5, 1.0
    return kind, p


def _add_mesh(sd, v, n, f, mats, tri_mat):
    """sd with a mesh and its materials (kind, 16 parameters) appended."""
    nv, m0 = sd.vertices.shape[0], sd.mat_type.shape[0]
    return dataclasses.replace(
        sd, vertices=np.concatenate([sd.vertices, v]), normals=np.concatenate([sd.normals, n]),
        indices=np.concatenate([sd.indices, (f + nv).astype(np.uint32)]),
        tri_material=np.concatenate([sd.tri_material, (tri_mat + m0).astype(np.uint32)]),
        tri_emission=np.concatenate([sd.tri_emission, np.full(f.shape[0], -1, np.int32)]),
        mat_type=np.concatenate([sd.mat_type, np.array([k for k, _ in mats], np.uint32)]),
        mat_params=np.concatenate([sd.mat_params, np.stack([p for _, p in mats])]))


def _vary(sd, rng):
    """Wall colours, light, spheres and camera of this seed."""
    mp = sd.mat_params.copy()
    diffuse = (sd.mat_type == scenes.MAT_DIFFUSE) & (mp[:, 0] > 0)
    mp[diffuse, 0:3] *= rng.uniform(0.8, 1.2, (int(diffuse.sum()), 3)).astype(np.float32)
    em = (sd.emission * rng.uniform(0.7, 1.3, (1, 3))).astype(np.float32)
    sph = sd.spheres
    if sph is not None:
        sph = sph.copy()
        sph[:, :3] += rng.uniform(-0.03, 0.03, sph[:, :3].shape).astype(np.float32)
    pos = tuple(float(x) for x in np.asarray(sd.camera.pos) + rng.uniform(-0.05, 0.05, 3))
    return dataclasses.replace(sd, mat_params=mp, emission=em, spheres=sph,
                               camera=dataclasses.replace(sd.camera, pos=pos))


def _mesh_box(level, rng, groups=64):
    v, n, f = _ball(level, 0.4, (0.0, -0.55, 0.0), rng)
    mats = [_material(scenes.MAT_CONDUCTOR, (1, 1, 1), alpha=a) for a in rng.uniform(0.05, 0.5, groups)]
    per = max(1, f.shape[0] // groups)
    grp = np.minimum(np.arange(f.shape[0]) // per, groups - 1)
    return _add_mesh(scenes.cornell_box(spheres=False), v, n, f, mats, grp)


def _mixed_box(level, rng):
    v, n, f = _ball(level, 0.35, (0.0, -0.3, 0.0), rng)
    mats = [_material(scenes.MAT_DIFFUSE, (0.6, 0.7, 0.5)),
            _material(scenes.MAT_CONDUCTOR, (0.9, 0.8, 0.7), alpha=float(rng.uniform(0.05, 0.5))),
            _material(scenes.MAT_DIELECTRIC, (1, 1, 1), (1, 1, 1), alpha=float(rng.uniform(0.05, 0.3)))]
    return _add_mesh(scenes.cornell_box(), v, n, f, mats, np.arange(f.shape[0]) * 3 // f.shape[0])


def _knot(half, env, rng):
    """2 half x half quads of a rough-glass torus knot under a sky map with a sun."""
    v, f, nrm = scenes.torus_knot(2 * half, half)
    v = (v + nrm * (0.006 * _ripple(v * 2.0, rng))[:, None]).astype(np.float32)
    if env not in _SKIES:
        _SKIES[env] = scenes.sky_envmap(env, env // 2, seed=5, sun_diameter_deg=0.5 if env > 1000 else 12)
    kind, p = _material(scenes.MAT_DIELECTRIC, (1, 1, 1), (1, 1, 1), alpha=float(rng.uniform(0.05, 0.2)))
    sky = (_SKIES[env] * rng.uniform(0.8, 1.2, 3)).astype(np.float32)
    return scenes.SceneDesc(
        vertices=v, normals=_smooth_normals(v.astype(np.float64), f), indices=f.astype(np.uint32),
        tri_material=np.zeros(f.shape[0], np.uint32), tri_emission=np.full(f.shape[0], -1, np.int32),
        mat_type=np.array([kind], np.uint32), mat_params=p[None], emission=np.zeros((0, 3), np.float32), env=sky,
        camera=scenes.Camera(pos=tuple(float(x) for x in np.array([0, 0, 3.0]) + rng.uniform(-0.05, 0.05, 3))))


def _desc(case, rng):
    kind = case["scene"]
    if kind == "cornell":
        return _vary(scenes.cornell_box(), rng)
    if kind == "mixed":
        return _vary(_mixed_box(case["level"], rng), rng)
    if kind == "mesh":
        return _vary(_mesh_box(case["level"], rng), rng)
    if kind == "knot":
        return _knot(case["level"], case["env"], rng)
    if kind == "fog":
        sd = scenes.cornell_fog(sigma_s=float(rng.uniform(0.3, 0.8)))
    else:
        sd = scenes.fog_ball_box(level=case["level"], sigma_s=float(rng.uniform(1.0, 3.0)))
    return _vary(sd, rng)


def _instance_sizes(case):
    """Film sizes, samples and subdivision levels of a batch's instances."""
    r = np.random.default_rng(case["salt"])
    lo = max(16, case["max_res"] // 8)
    for i in range(case["instances"]):
        rx, ry = (int(round(math.exp(r.uniform(math.log(lo), math.log(case["max_res"]))))) for _ in range(2))
        yield rx, ry, int(r.integers(1, case["max_spp"] + 1)), int(r.integers(2, case["max_level"] + 1)), bool(
            r.integers(0, 2))


def _instance(level, is_diffuse, rng):
    v, n, f = _ball(level, 0.42, (0.0, -0.5, 0.0), rng)
    albedo = tuple(rng.uniform(0.2, 0.9, 3))
    mat = (_material(scenes.MAT_DIFFUSE, albedo) if is_diffuse
           else _material(scenes.MAT_CONDUCTOR, albedo, alpha=float(rng.uniform(0.05, 0.5))))
    return _vary(_add_mesh(scenes.cornell_box(spheres=False), v, n, f, [mat], np.zeros(f.shape[0], np.int64)), rng)


def _rays(n, rng):
    """Rays from a shell around the scene's middle into the box, unit directions."""
    o = rng.uniform(-0.9, 0.9, (n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d, np.full((n, 1), np.inf)], 1).astype(np.float32)


# ---------------------------------------------------------------- protocol ---
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ctx = _context(case)
    kind = case["kind"]
    if kind == "batch":
        held, cams, prms, out = [], [], [], []
        for rx, ry, spp, level, is_diffuse in _instance_sizes(case):
            sd = _instance(level, is_diffuse, rng)
            held.append(g.Scene(sd, ctx))
            cams.append(dataclasses.replace(sd.camera, res_x=rx, res_y=ry))
            prms.append(scenes.RenderParams(spp, case["depth"], case["rr"], case["sampler"]))
            out.append(torch.empty((ry, rx, 3), dtype=torch.float32, pin_memory=True).numpy())
        ctx.set_batch_config(paths_in_flight=case["pool"])
        return dict(kind=kind, ctx=ctx, scenes=held, cams=cams, prms=prms, out=out)
    if kind == "rays":
        return dict(kind=kind, scene=g.Scene(_desc(case, rng), ctx), rays=_rays(case["rays"], rng),
                    any_hit=case["any_hit"])
    if kind == "adjoint":
        groups = case["groups"]
        hidden = scenes.inverse_params(groups=groups, seed=seed)
        start = scenes.perturb_params(hidden, seed=seed + 1)
        sd = scenes.inverse_box(start, level=case["level"], res=case["res_x"], spp=case["spp"], max_depth=case["depth"],
                                rr_depth=case["depth"])
        sd.camera = dataclasses.replace(sd.camera, res_x=case["res_x"], res_y=case["res_y"])
        sd.params = dataclasses.replace(sd.params, sampler=case["sampler"])
        leaf = [torch.tensor(x, dtype=torch.float64, device="cuda", requires_grad=True)
                for x in (start.albedo, start.alpha, start.radiance)]
        target = torch.rand((case["res_y"], case["res_x"], 3), dtype=torch.float64, device="cuda",
                            generator=torch.Generator("cuda").manual_seed(seed))
        return dict(kind=kind, renderer=diff.DiffRenderer(ctx, sd), leaf=leaf, target=target)
    sd = _desc(case, rng)
    film = g.Film(case["res_x"], case["res_y"])
    cam = sd.camera
    camera = g.PinHoleCamera(film, cam.pos, cam.look_at, cam.up, cam.fovy, cam.film_distance)
    if kind == "path":
        integrator = g.GpuPathTracing(case["spp"], case["depth"], case["rr"], sampler=case["sampler"])
    elif kind == "volume":
        integrator = g.VolPathTracing(case["spp"], case["depth"], sampler=case["sampler"], equal_angular=case["equi"])
    else:
        integrator = g.LightTracing(case["depth"], case["spp"], sampler=case["sampler"])
    return dict(kind=kind, renderer=g.Renderer(g.Scene(sd, ctx), camera, integrator))


def run(state):
    kind = state["kind"]
    if kind == "batch":
        return state["ctx"].render_batch(state["scenes"], state["cams"], state["prms"], out=state["out"])
    if kind == "rays":
        return state["scene"].intersect(state["rays"], any_hit=state["any_hit"])
    if kind == "adjoint":
        leaf = state["leaf"]
        img = diff.PathReplayRender.apply(*leaf, state["renderer"])
        grads = torch.autograd.grad(diff.l2_loss(img, state["target"]), leaf)
        return [img.detach(), *grads]
    return state["renderer"].Render().image


def _triangles(case):
    return {"cornell": 12, "fog": 14, "fog_ball": 12 + 20 * 4 ** case.get("level", 0),
            "mixed": 12 + 20 * 4 ** case.get("level", 0), "mesh": 12 + 20 * 4 ** case.get("level", 0),
            "knot": 4 * case.get("level", 0) ** 2}[case["scene"]]


# One triangle of the scene as the tracer reads it: three positions, three
# normals, a material. One bounce of a path: a tree of the scene's triangles
# walked to one leaf twice (the path's ray, its shadow ray) at a box test of
# about 24 operations a level, a triangle test of about 60 each, and about 300
# operations to sample the light, the surface and the next direction.
TRIANGLE_BYTES = 3 * 12 + 3 * 12 + 8


def _bounce_flops(tris):
    return 2 * (24 * math.log2(tris + 2) + 60) + 300


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for rx, ry, spp, level, _ in _instance_sizes(case):
            tris = 12 + 20 * 4 ** level
            b += TRIANGLE_BYTES * tris + 12 * rx * ry
            f += rx * ry * spp * min(4, case["depth"]) * _bounce_flops(tris)
        return dict(bytes=b, flops=f)
    if kind == "rays":
        tris = _triangles(case)
        return dict(bytes=TRIANGLE_BYTES * tris + case["rays"] * (28 + 16),
                    flops=case["rays"] * (24 * math.log2(tris + 2) + 60))
    px = case["res_x"] * case["res_y"]
    if kind == "adjoint":
        tris = 18 + 20 * 4 ** case["level"]
        return dict(bytes=TRIANGLE_BYTES * tris + px * (24 + 24 + 12 * case["spp"]),
                    flops=2 * px * case["spp"] * min(4, case["depth"]) * _bounce_flops(tris))
    tris = _triangles(case)
    bounces = min(4, case["depth"]) if case["scene"] != "knot" else 1.3
    env = case.get("env", 0) ** 2 // 2 * 16
    return dict(bytes=TRIANGLE_BYTES * tris + env + 12 * px, flops=px * case["spp"] * bounces * _bounce_flops(tris))


def exact(case, seed):
    """Closest hits in 64 bits by testing every triangle; images and gradients
    are sums over sampled paths that have no value of this kind."""
    if case["kind"] != "rays" or case["any_hit"] or case["scene"] != "mesh":
        return None
    if case["rays"] * _triangles(case) > 8e9:
        return None
    rng = np.random.default_rng(seed)
    sd = _desc(case, rng)
    rays = torch.from_numpy(_rays(case["rays"], rng)).cuda().double()
    p = torch.from_numpy(sd.vertices[sd.indices.astype(np.int64)]).cuda().double()
    p0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    plane = (p0 * nrm).sum(1)
    # barycentric weights of vertices 1 and 2 are affine in the hit point
    nn = (nrm * nrm).sum(1, keepdim=True)
    wu, wv = torch.linalg.cross(e2, nrm) / nn, torch.linalg.cross(nrm, e1) / nn
    cu, cv = (p0 * wu).sum(1), (p0 * wv).sum(1)
    ts, us, vs = [], [], []
    step = max(1, int(4e7) // p.shape[0])
    for r in rays.split(step):
        o, d = r[:, :3], r[:, 3:6]
        t = (plane[None] - o @ nrm.T) / (d @ nrm.T)
        u = o @ wu.T + t * (d @ wu.T) - cu
        v = o @ wv.T + t * (d @ wv.T) - cv
        t = torch.where((t >= 0) & (u >= 0) & (v >= 0) & (u + v <= 1), t, torch.inf)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        zero = torch.zeros_like(best)
        ts.append(torch.where(hit, best, zero))
        us.append(torch.where(hit, u.gather(1, k[:, None])[:, 0], zero))
        vs.append(torch.where(hit, v.gather(1, k[:, None])[:, 0], zero))
    return [None, torch.cat(ts), torch.cat(us), torch.cat(vs)]
