"""The work that is timed: builds and traces as a program that uses the package asks for them.

A case is a dict of plain values. ``listed()`` gives the fixed ones, ``draw(rng)`` one more of the same ranges,
``prepare`` what a program has in hand before the call (inputs on the GPU, and the BVH or plan that it keeps),
``run`` one pass through the public entry points, ``work`` what a pass cannot do without, ``exact`` its results in 64
bits. Scenes have the shapes of ``diplodocus_b200.scenes`` (the open box with a sphere, the displaced sphere, the
log-normal soup), made on the GPU.
"""
from __future__ import annotations

import math

import torch

from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S
from diplodocus_b200.autograd import closest_hit_tuv

K_EPSILON = 1e-6
K_INFINITY = 3.4028234663852886e38
ROOM_CAMERA = S.SMALL_CAMERA
SPHERE_CAMERA = S.DIFF_CAMERA
# triangles of the open box that the room's lights are: the two of its ceiling
ROOM_AREA_LIGHTS = (2, 3)
ROOM_POINT_LIGHTS = ((0.3, 0.35, 0.2),)


def _case(kind, scene, triangles, rays, **options):
    """A case with every field: the options that a kind does not read keep these values."""
    case = dict(kind=kind, scene=scene, triangles=triangles, rays=rays, width=0, height=0, accel="ploc",
                layout="binary", clustering="hploc", leaf_test="ref_mt", split=0, radius=16, leaf=4, culling=False,
                coherent=False, area_samples=0, point_lights=False, meshes=0)
    case.update(options)
    return case


def listed():
    return [
        # an interactive preview: one small frame of a small scene, where launches and host work are the cost
        dict(_case("frame", "room", 3978, 0, width=64, height=64), name="frame_64"),
        # a renderer's frame with direct light: primary and bounce rays, area-light and point-light shadow rays
        dict(_case("frame", "room", 3978, 0, width=512, height=512, area_samples=4, point_lights=True),
             name="frame_512_lights"),
        # a small dynamic scene, rebuilt and traced every frame
        dict(_case("rebuild", "room", 3978, 16384), name="rebuild_small"),
        # a detailed deforming mesh, rebuilt and seen by a camera
        dict(_case("rebuild", "sphere", 1046528, 65536), name="rebuild_sphere_1m"),
        # a large scene with triangles of very different sizes, loaded once: extended codes and pre-splitting
        dict(_case("rebuild", "soup", 16777216, 262144, accel="ploc_emc", split=40), name="rebuild_soup_16m"),
        # a mesh of odd size with oriented bounding slabs
        dict(_case("rebuild", "sphere", 250020, 100003, accel="ploc_emc_sobb"), name="rebuild_sobb_250k"),
        # many rays of a renderer's sample loop against one detailed mesh
        dict(_case("trace", "sphere", 1046528, 4194304), name="trace_sphere_4m"),
        # incoherent rays through the large scene, sorted by the library
        dict(_case("trace", "soup", 16777216, 16777216, accel="ploc_emc", split=40, coherent=True),
             name="trace_soup_16m"),
        # the compressed layout, for scenes whose nodes have to stay small
        dict(_case("trace", "soup", 2000003, 2097152, layout="wide8_q8", split=40, coherent=True),
             name="trace_wide_2m"),
        # occlusion queries between points of a scene, watertight and with culling, in the order they come
        dict(_case("occlusion", "soup", 300007, 1000003, leaf_test="watertight", culling=True, split=20),
             name="occlusion_1m"),
        # many meshes of very different sizes, rebuilt by one captured plan and each traced
        dict(_case("batch", "sphere", 100000, 4096, meshes=32), name="batch_32"),
        # a fitting step: depth and barycentrics of a camera's hits, and their gradients
        dict(_case("diff", "sphere", 65024, 0, width=1024, height=1024), name="diff_1m"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _leaf(rng, form):
    """The 8-wide layout takes leaves of at most 5."""
    return rng.choice((2, 4, 5 if form == "wide" else 8))


def draw(rng):
    kind = rng.choice(("frame", "rebuild", "rebuild", "trace", "trace", "occlusion", "batch", "diff"))
    accel = rng.choice(("ploc", "ploc_emc"))
    leaf_test = rng.choice(("ref_mt", "ref_mt", "watertight"))
    if kind == "frame":
        w = _log_uniform(rng, 48, 640)
        h = max(32, int(w * rng.uniform(0.5, 1.0)))
        return _case(kind, "room", _log_uniform(rng, 1000, 200000), 0, width=w, height=h, accel=accel,
                     area_samples=rng.choice((0, 1, 4)), point_lights=rng.random() < 0.5,
                     layout=rng.choice(("binary", "binary", "wide8_q8")))
    if kind == "rebuild":
        scene = rng.choice(("room", "sphere", "soup"))
        n = _log_uniform(rng, 1000, 8000000 if scene == "soup" else 1000000)
        form = rng.choice(("aabb", "aabb", "sobb", "wide"))
        return _case(kind, scene, n, _log_uniform(rng, 4096, 262144), accel=accel + ("_sobb" if form == "sobb" else ""),
                     layout="wide8_q8" if form == "wide" else "binary", leaf_test=leaf_test,
                     clustering=rng.choice(("hploc", "hploc", "ploc")), radius=rng.choice((8, 10, 16)),
                     leaf=_leaf(rng, form), split=rng.choice((20, 40)) if scene == "soup" else 0)
    if kind == "trace":
        scene = rng.choice(("room", "sphere", "soup"))
        form = rng.choice(("aabb", "aabb", "sobb", "wide"))
        n = _log_uniform(rng, 1000, 4000000 if scene == "soup" else 1000000)
        return _case(kind, scene, n, _log_uniform(rng, 1000, 4194304), accel=accel + ("_sobb" if form == "sobb" else ""),
                     layout="wide8_q8" if form == "wide" else "binary", leaf_test=leaf_test, leaf=_leaf(rng, form),
                     culling=rng.random() < 0.25, split=rng.choice((20, 40)) if scene == "soup" else 0,
                     coherent=scene == "soup")
    if kind == "occlusion":
        scene = rng.choice(("room", "sphere", "soup"))
        return _case(kind, scene, _log_uniform(rng, 1000, 1000000), _log_uniform(rng, 1000, 4194304), accel=accel,
                     layout=rng.choice(("binary", "binary", "wide8_q8")), leaf_test=leaf_test,
                     culling=rng.random() < 0.5, split=20 if scene == "soup" else 0)
    if kind == "batch":
        return _case(kind, "sphere", _log_uniform(rng, 5000, 200000), _log_uniform(rng, 1000, 8192),
                     meshes=_log_uniform(rng, 4, 64), accel=accel, clustering=rng.choice(("hploc", "ploc")))
    w = _log_uniform(rng, 128, 1024)
    return _case(kind, "sphere", _log_uniform(rng, 5000, 100000), 0, width=w,
                 height=max(64, int(w * rng.uniform(0.5, 1.0))), leaf_test=leaf_test, accel=accel)


# -- scenes and rays on the GPU -------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _sphere_size(triangles):
    """(nu, nv) of the UV sphere with nu = 2 nv whose 2 nu (nv - 1) triangles come nearest to the number asked for."""
    nv = max(3, round(math.sqrt(triangles / 4.0 + 0.25) + 0.5))
    return 2 * nv, nv


def _sphere(triangles, g, radius=1.0, center=(0.0, 0.0, 0.0), displacement=0.05):
    """A UV sphere, its radius displaced by four octaves of smooth noise: (N, 3, 3) float32, ring by ring."""
    nu, nv = _sphere_size(triangles)
    f64 = dict(dtype=torch.float64, device="cuda")
    theta = (torch.arange(1, nv, **f64) * (math.pi / nv))[:, None]
    phi = (torch.arange(nu, **f64) * (2.0 * math.pi / nu))[None, :]
    ring = torch.stack([theta.sin() * phi.cos(), theta.cos() * torch.ones_like(phi), theta.sin() * phi.sin()], dim=-1)
    pole = torch.tensor([[0.0, 1.0, 0.0]], **f64)
    dirs = torch.cat([pole, ring.reshape(-1, 3), -pole])
    r = torch.full((dirs.shape[0],), radius, **f64)
    if displacement:
        noise = torch.zeros_like(r)
        for octave in range(4):
            k = (8 << octave) + 1
            grid = torch.rand((1, 1, k, k, k), generator=g, **f64) * 2.0 - 1.0
            at = dirs.reshape(1, 1, 1, -1, 3)
            noise += 0.5 ** octave * torch.nn.functional.grid_sample(grid, at, align_corners=True).reshape(-1)
        r = r * (1.0 + displacement * noise / 1.875)
    verts = (dirs * r[:, None] + torch.tensor(center, **f64)).to(torch.float32)
    seg = torch.arange(nu, device="cuda")
    nxt = (seg + 1) % nu
    rings = 1 + torch.arange(nv - 1, device="cuda")[:, None] * nu
    a, b = rings[:-1] + seg, rings[:-1] + nxt
    c, d = rings[1:] + seg, rings[1:] + nxt
    last = verts.shape[0] - 1
    idx = torch.cat([
        torch.stack([torch.zeros_like(seg), rings[0] + nxt, rings[0] + seg], dim=1),
        torch.cat([torch.stack([a, b, d], dim=2), torch.stack([a, d, c], dim=2)], dim=1).reshape(-1, 3),
        torch.stack([torch.full_like(seg, last), rings[-1] + seg, rings[-1] + nxt], dim=1),
    ])
    return verts[idx].contiguous()


def _room(triangles, g):
    """The open box with a sphere in it, its centre moved by the seed."""
    shift = (torch.rand(3, generator=g, device="cuda") - 0.5).mul(0.3).tolist()
    center = (shift[0], shift[1] - 0.2, shift[2] - 0.1)
    return torch.cat([torch.from_numpy(S.open_box()).cuda(), _sphere(triangles - 10, g, 0.25, center, 0.0)])


def _soup(triangles, g):
    """Uniform centroids, log-normal edge lengths, a fifth of the triangles skinny (1:50), random orientation. The
    lengths shrink with the cube root of the count as if the soup were cut out of the 16M one, so that every size has
    its density."""
    dev = dict(device="cuda", generator=g)
    n = triangles
    scale = (16777216 / n) ** (1.0 / 3.0)
    ell = torch.exp(-6.0 + 1.5 * torch.randn(n, **dev)) * scale
    short = torch.where(torch.rand(n, **dev) < 0.2, ell / 50.0, ell)
    phi = torch.deg2rad(30.0 + 120.0 * torch.rand(n, **dev))
    e1 = torch.nn.functional.normalize(torch.randn((n, 3), **dev), dim=1)
    side = torch.nn.functional.normalize(torch.linalg.cross(e1, torch.randn((n, 3), **dev)), dim=1)
    p1 = e1 * ell[:, None]
    p2 = e1 * (short * phi.cos())[:, None] + side * (short * phi.sin())[:, None]
    pts = torch.stack([torch.zeros_like(p1), p1, p2], dim=1)
    return pts - pts.mean(dim=1, keepdim=True) + torch.rand((n, 1, 3), **dev)


def _scene(case, g):
    return {"room": _room, "sphere": _sphere, "soup": _soup}[case["scene"]](case["triangles"], g)


def _unit(n, g):
    return torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)


def _rays(case, n, g):
    """Rays as the scene's users cast them: from around the sphere inward, from random points of the soup, and from
    the room's camera side into the room, pixel by pixel."""
    rays = torch.empty((n, 8), device="cuda")
    if case["scene"] == "room":
        w = max(1, math.isqrt(n))
        i = torch.arange(n, device="cuda")
        x, y = (i % w) / w - 0.5, (i // w) / w - 0.5
        shift = 0.02 * torch.rand(3, generator=g, device="cuda")
        rays[:, 0:3] = torch.tensor(ROOM_CAMERA["cam_pos"], device="cuda") + shift
        rays[:, 4:7] = torch.nn.functional.normalize(torch.stack([x, -y, torch.full_like(x, -1.0)], dim=1), dim=1)
    elif case["scene"] == "sphere":
        p, d = _unit(n, g), _unit(n, g)
        rays[:, 0:3] = 3.0 * p
        rays[:, 4:7] = torch.where((p * d).sum(1, keepdim=True) > 0, -d, d)
    else:
        rays[:, 0:3] = torch.rand((n, 3), generator=g, device="cuda")
        rays[:, 4:7] = _unit(n, g)
    rays[:, 3] = K_EPSILON
    rays[:, 7] = K_INFINITY
    return rays


def _camera(g):
    """The room's camera, moved a little by the seed (pixels of the centred one lie on the walls' diagonals)."""
    x, y = (torch.rand(2, generator=g, device="cuda") * 0.04 - 0.02).tolist()
    return dict(ROOM_CAMERA, cam_pos=(x, y, ROOM_CAMERA["cam_pos"][2]))


def _segments(case, n, g):
    """Rays of occlusion queries: as ``_rays``, ending at a distance of the scene's scale."""
    rays = _rays(case, n, g)
    rays[:, 7] = torch.rand(n, generator=g, device="cuda") * {"room": 2.0, "sphere": 4.0, "soup": 0.3}[case["scene"]]
    return rays


# -- preparation and passes -----------------------------------------------------------------------------------
def _config(case):
    return A.AccelerationStructureConfig(
        acceleration_structure_type=A.parse_acceleration_structure_type(case["accel"]), layout=case["layout"],
        clustering=case["clustering"], leaf_test=case["leaf_test"], split_budget=case["split"],
        nn_search_radius=case["radius"], max_triangles_per_leaf=case["leaf"])


def _mesh_sizes(case):
    """Triangles of a batch's meshes: spread over the logarithm from a fiftieth of the largest up to it."""
    m, largest = case["meshes"], case["triangles"]
    return [max(24, round(largest * 50.0 ** (-k / max(1, m - 1)))) for k in range(m)]


def prepare(case, seed):
    g = _generator(seed)
    state = dict(case=case, seed=seed)
    kind = case["kind"]
    if kind == "batch":
        meshes = [_sphere(n, g) for n in _mesh_sizes(case)]
        state["rays"] = [_rays(case, case["rays"], g) for _ in meshes]
        state["plan"] = A.BuildPlan(_config(case), meshes)
        state["meshes"] = meshes
        return state
    state["triangles"] = _scene(case, g)
    state["bvh"] = A.GpuPlocBvh()
    if kind == "rebuild":
        state["rays"] = _rays(case, case["rays"], g)
        return state
    state["bvh"].Build(_config(case), A.Stats(), state["triangles"])
    if kind == "trace":
        state["rays"] = _rays(case, case["rays"], g)
    elif kind == "occlusion":
        state["rays"] = _segments(case, case["rays"], g)
    elif kind == "frame":
        state["camera"], state["lights"] = _camera(g), None
        if case["area_samples"] or case["point_lights"]:
            state["lights"] = A.Lights(ROOM_AREA_LIGHTS if case["area_samples"] else (), max(1, case["area_samples"]),
                                       ROOM_POINT_LIGHTS if case["point_lights"] else ())
    else:
        c = SPHERE_CAMERA
        rays = A.generate_pinhole_rays(c["cam_pos"], c["cam_dir"], c["cam_up"], c["fov"], c["far"], case["width"],
                                       case["height"])
        leaf = lambda t: t.clone().contiguous().requires_grad_(True)  # noqa: E731
        state["inputs"] = [leaf(state["triangles"][:, k]) for k in range(3)] + [leaf(rays[:, 0:3]), leaf(rays[:, 4:7])]
        state["far"] = c["far"]
        state["upstream"] = [torch.randn(rays.shape[0], generator=g, device="cuda") for _ in range(3)]
    return state


def _records(hits):
    return dict(prim=hits.prim, t=hits.t, u=hits.u, v=hits.v)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    stats = A.Stats()
    if kind == "frame":
        out = A.trace_frame(state["bvh"], state["camera"], case["width"], case["height"], state["seed"] & 0xFFFF,
                            lights=state["lights"])
        result = dict(rays=out[0], hits=_records(out[1]), bounce=out[2], bounce_hits=_records(out[3]))
        if state["lights"] is not None:
            result.update(shadow=out[4], occluded=out[5])
        return result
    if kind == "rebuild":
        state["bvh"].Build(_config(case), stats, state["triangles"])
        return _records(state["bvh"].Intersect(stats, state["rays"]))
    if kind == "trace":
        return _records(state["bvh"].Intersect(stats, state["rays"], backface_culling=case["culling"],
                                               coherent_order=case["coherent"]))
    if kind == "occlusion":
        return state["bvh"].IntersectAny(stats, state["rays"], backface_culling=case["culling"])
    if kind == "batch":
        state["plan"].launch()
        hits = [b.Intersect(stats, r) for b, r in zip(state["plan"].bvhs(), state["rays"])]
        raw = torch.cat([h.raw for h in hits])
        f = raw.view(torch.float32)
        return dict(prim=raw[:, 0], t=f[:, 1], u=f[:, 2], v=f[:, 3])
    t, u, v, prim = closest_hit_tuv(*state["inputs"], state["bvh"], tmax=state["far"], leaf_test=case["leaf_test"])
    grads = torch.autograd.grad((t, u, v), state["inputs"], state["upstream"])
    return dict(t=t, u=u, v=v, prim=prim, dv=list(grads[:3]), dorigin=grads[3], ddirection=grads[4])


def work(case):
    """Bytes: the vertices that a build reads and the leaf triangles and nodes that it has to write (100 bytes a
    triangle in all), rays and records; a trace alone reads its scene's vertices once. Operations: the box tests of a
    balanced tree's path for every ray."""
    kind, n = case["kind"], case["triangles"]
    rays, levels = case["rays"], max(1.0, math.log2(n))
    if kind == "batch":
        sizes = _mesh_sizes(case)
        rays *= len(sizes)
        return dict(bytes=100 * sum(sizes) + 48 * rays, flops=rays * levels * 24)
    if kind == "rebuild":
        return dict(bytes=100 * n + 48 * rays, flops=rays * levels * 24)
    if kind == "trace":
        return dict(bytes=36 * n + 48 * rays, flops=rays * levels * 24)
    if kind == "occlusion":
        return dict(bytes=36 * n + 33 * rays, flops=rays * levels * 24)
    pixels = case["width"] * case["height"]
    if kind == "diff":  # rays, records, three upstream values, gradients of rays and vertices
        return dict(bytes=72 * n + pixels * (32 + 16 + 12 + 24), flops=pixels * (levels * 24 + 200))
    shadow = pixels * (2 * case["area_samples"] + int(case["point_lights"]))
    return dict(bytes=36 * n + pixels * 2 * 48 + shadow * 33, flops=(2 * pixels + shadow) * levels * 24)


# -- 64-bit results -------------------------------------------------------------------------------------------
def _closest(tris, rays, culling, cull_det):
    """Closest hits in 64 bits over all pairs: the side products of Plücker coordinates are matrix products. Ties go
    to the lowest index. ``cull_det``: the reference leaf test refuses |det| < 1e-6."""
    tris, rays = tris.double(), rays.double()
    v0, v1, v2 = tris.unbind(1)
    o, d = rays[:, 0:3], rays[:, 4:7]
    cross = torch.linalg.cross
    line = torch.cat([d, cross(o, d)], dim=1)
    edge = lambda a, b: torch.cat([cross(a, b), b - a], dim=1).T.contiguous()  # noqa: E731
    e12, e20, e01 = edge(v1, v2), edge(v2, v0), edge(v0, v1)
    normal = cross(v1 - v0, v2 - v0)
    plane = torch.cat([-normal, (normal * v0).sum(1, keepdim=True)], dim=1).T.contiguous()
    point = torch.cat([o, torch.ones_like(o[:, :1])], dim=1)
    nt = normal.T.contiguous()
    prim = torch.full((len(rays),), -1, dtype=torch.int64, device=rays.device)
    step = max(1, (1 << 27) // len(tris))
    for a in range(0, len(rays), step):
        s = slice(a, a + step)
        w0, w1, w2 = line[s] @ e12, line[s] @ e20, line[s] @ e01
        inside = ((w0 >= 0) & (w1 >= 0) & (w2 >= 0)) | ((w0 <= 0) & (w1 <= 0) & (w2 <= 0))
        del w0, w1, w2
        det = d[s] @ nt
        if cull_det:
            inside &= det.abs() >= 1e-6
        if culling:
            inside &= det < 0
        t = (point[s] @ plane) / det
        t = torch.where(inside & (t > rays[s, 3:4]) & (t < rays[s, 7:8]), t, math.inf)
        near, at = t.min(dim=1)
        prim[s] = torch.where(near < math.inf, at, -1)
        del det, t, inside
    return prim


def _tuv(v0, v1, v2, o, d):
    """Möller-Trumbore of one triangle a ray."""
    cross = torch.linalg.cross
    e1, e2, s = v1 - v0, v2 - v0, o - v0
    p, q = cross(d, e2), cross(s, e1)
    det = (e1 * p).sum(1)
    return (e2 * q).sum(1) / det, (s * p).sum(1) / det, (d * q).sum(1) / det


def _exact_records(tris, rays, case):
    prim = _closest(tris, rays, case["culling"], case["leaf_test"] == "ref_mt")
    hit = prim >= 0
    tri, r = tris[prim.clamp(min=0)].double(), rays.double()
    t, u, v = _tuv(tri[:, 0], tri[:, 1], tri[:, 2], r[:, 0:3], r[:, 4:7])
    zero = torch.zeros_like(t)
    return dict(prim=None, t=torch.where(hit, t, math.inf), u=torch.where(hit, u, zero), v=torch.where(hit, v, zero))


def _pinhole(camera, width, height):
    """The frame's primary rays in 64 bits."""
    vec = lambda k: torch.tensor(camera[k], dtype=torch.float64, device="cuda")  # noqa: E731
    fwd, up = vec("cam_dir"), vec("cam_up")
    right = torch.nn.functional.normalize(torch.linalg.cross(fwd, up), dim=0)
    gw = 2.0 * math.tan(camera["fov"] / 2.0)
    gh = gw * height / width
    i = torch.arange(width * height, device="cuda")
    x, y = (i % width).double()[:, None], (i // width).double()[:, None]
    d = fwd - right * gw / 2 + up * gh / 2 + right * (gw / (width - 1)) * x - up * (gh / (height - 1)) * y
    rays = torch.empty((width * height, 8), dtype=torch.float64, device="cuda")
    rays[:, 0:3], rays[:, 3], rays[:, 7] = vec("cam_pos"), K_EPSILON, camera["far"]
    rays[:, 4:7] = torch.nn.functional.normalize(d, dim=1)
    return rays


def exact(case, seed):
    kind = case["kind"]
    pixels = case["width"] * case["height"]
    pairs = case["triangles"] * (pixels or case["rays"]) * max(1, case["meshes"])
    if kind == "occlusion" or pairs > 1.2e11:  # flags only, or too many pairs to go through
        return None
    g = _generator(seed)
    if kind == "batch":
        meshes = [_sphere(n, g) for n in _mesh_sizes(case)]
        parts = [_exact_records(m, _rays(case, case["rays"], g), case) for m in meshes]
        return dict(prim=None, **{k: torch.cat([p[k] for p in parts]) for k in "tuv"})
    tris = _scene(case, g)
    if kind in ("rebuild", "trace"):
        return _exact_records(tris, _rays(case, case["rays"], g), case)
    if kind == "frame":  # what follows the primary hits is drawn at random by the library's own hash
        rays = _pinhole(_camera(g), case["width"], case["height"])
        return dict(rays=rays, hits=_exact_records(tris, rays, case), bounce=None, bounce_hits=None)
    camera = _pinhole(SPHERE_CAMERA, case["width"], case["height"]).float()
    prim = _closest(tris, camera, False, case["leaf_test"] == "ref_mt")
    hit = prim >= 0
    inputs = [x.double().requires_grad_(True) for x in (*tris.unbind(1), camera[:, 0:3], camera[:, 4:7])]
    at = prim[hit]
    tuv = _tuv(*(x[at] for x in inputs[:3]), *(x[hit] for x in inputs[3:]))
    upstream = [torch.randn(len(camera), generator=g, device="cuda").double()[hit] for _ in range(3)]
    grads = torch.autograd.grad(tuv, inputs, upstream)
    whole = [torch.full((len(camera),), miss, dtype=torch.float64, device="cuda") for miss in (math.inf, 0.0, 0.0)]
    t, u, v = (w.masked_scatter(hit, x.detach()) for w, x in zip(whole, tuv))
    return dict(t=t, u=u, v=v, prim=None, dv=list(grads[:3]), dorigin=grads[3], ddirection=grads[4])
