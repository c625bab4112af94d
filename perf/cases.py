"""Workloads that are timed: the calls a renderer host makes of this library.

  trace      device-resident rays against one displaced icosphere
             (GpuAccelerator.trace_closest / trace_any)
  host       the drop-in batch call on host rays (GpuAccelerator.intersect_batch)
  instances  device-resident rays against a two-level scene
             (InstancedAccelerator.trace_closest)
  render     a diffuse box scene (Renderer.render, graph-captured waves)
  materials  the box scene with every material, corrected MIS, first-hit albedo
             and normal films
  field      the two-level scene under a sky light, mixed materials and a
             homogeneous medium box
  batch      several scenes through one BatchRenderer
  adjoint    forward render and path-replay adjoint of the textured box scene

listed() names the cases, draw() makes more of the same ranges, prepare() builds
what a host program holds before the call (scene handles, renderers, films and
the inputs of the given seed), run() is one pass, work() the bytes and operations
that no implementation can do without, tolerance() how far another correct
implementation at the same precision may be off, exact() the same result in 64
bits by plain torch, from the definitions of the algorithms.
"""
import functools
import math

import numpy as np
import torch

from gonzales_b200 import _ffi as F
from gonzales_b200 import adjoint as A
from gonzales_b200 import scenes
from gonzales_b200.accel import BatchRenderer, GpuAccelerator, InstancedAccelerator, Renderer

DEV = "cuda"
MEDIUM = dict(box_min=(-10.0, -6.0, -10.0), box_max=(10.0, 6.0, 10.0), sigma_a=(0.05,) * 3, sigma_s=(0.2,) * 3, g=0.0)


def listed():
    return [
        # one 64 x 64 tile's camera rays, as a tile renderer issues them: a few
        # microseconds of work behind one launch
        dict(name="tile_closest", kind="trace", subdiv=5, rays="camera", query="closest", width=64, height=64),
        # the camera half of the ray-cast workload: 8M pinhole rays, 1.31M triangles
        dict(name="camera_closest", kind="trace", subdiv=8, rays="camera", query="closest", width=4096, height=2048),
        # its incoherent half: what diffuse bounces of a path tracer look like
        dict(name="scatter_closest", kind="trace", subdiv=8, rays="scatter", query="closest", count=8388608),
        # shadow rays of a large frame, a count that fills no block or chunk evenly
        dict(name="scatter_any", kind="trace", subdiv=8, rays="scatter", query="any", count=4000037),
        # the reference host's call: about 1e6 rays a batch from and to host arrays
        dict(name="host_batch", kind="host", subdiv=7, count=1000000),
        # rays through 4096 instances of 16 meshes of 50,000 triangles
        dict(name="instances_closest", kind="instances", count=2097152),
        # an interactive preview: one small frame, few samples
        dict(name="render_preview", kind="render", width=64, height=64, spp=4, depth=5, rr=3),
        # the plain path tracer's box scene frame
        dict(name="render_box", kind="render", width=256, height=256, spp=16, depth=5, rr=3),
        # every BSDF, both MIS strategies, AOV films, a frame of ragged size
        dict(name="render_materials", kind="materials", width=250, height=187, spp=16, depth=8, rr=2),
        # the full integrator: instances, sky light, layered materials, medium
        dict(name="render_field", kind="field", width=640, height=360, spp=16, depth=8, rr=2),
        # scenes of uneven size and film through shared waves
        dict(name="render_batch", kind="batch", scenes=8, spp=16, depth=6, rr=2),
        # one optimisation step of the albedo textures: forward and adjoint
        dict(name="adjoint_box", kind="adjoint", side=256, spp=16, depth=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "host", "instances", "render", "render", "materials", "field", "batch",
                       "adjoint"])
    if kind == "trace":
        c = dict(kind=kind, subdiv=rng.randint(3, 8), rays=rng.choice(["camera", "scatter"]),
                 query=rng.choice(["closest", "any"]))
        if c["rays"] == "camera":
            c.update(width=_log(rng, 32, 4096), height=_log(rng, 32, 2048))
        else:
            c.update(count=_log(rng, 1000, 8388608))
        return c
    if kind == "host":
        return dict(kind=kind, subdiv=rng.randint(4, 7), count=_log(rng, 2000, 1000000))
    if kind == "instances":
        return dict(kind=kind, count=_log(rng, 20000, 2097152))
    if kind == "render":
        return dict(kind=kind, width=_log(rng, 24, 256), height=_log(rng, 24, 256), spp=rng.choice([1, 2, 4, 8, 16]),
                    depth=rng.randint(2, 5), rr=rng.randint(2, 3))
    if kind == "materials":
        return dict(kind=kind, width=_log(rng, 40, 250), height=_log(rng, 40, 187), spp=rng.choice([1, 4, 16]),
                    depth=rng.randint(3, 8), rr=2)
    if kind == "field":
        return dict(kind=kind, width=_log(rng, 80, 640), height=_log(rng, 60, 360), spp=rng.choice([1, 4, 16]),
                    depth=rng.randint(4, 8), rr=2)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 8), spp=rng.choice([1, 4, 16]), depth=rng.randint(3, 6), rr=2)
    return dict(kind=kind, side=_log(rng, 40, 256), spp=rng.choice([1, 2, 4, 16]), depth=rng.randint(2, 5))


# ---------------------------------------------------------------- inputs

# Geometry of a case is the scene file a program loads: it is built once per
# process; views, rays, sample sequences and textures change with the seed.


@functools.lru_cache(maxsize=None)
def _sphere(subdiv):
    return scenes.raycast_scene(subdiv=subdiv).build()


@functools.lru_cache(maxsize=None)
def _field():
    return scenes.instanced_scene(mixed=True)


@functools.lru_cache(maxsize=None)
def _sky():
    return scenes.sky_map()


@functools.lru_cache(maxsize=None)
def _batch(n):
    return [(sb.build(), side) for sb, side in scenes.batch_workload(n, 0xC3, tri_lo=1000, tri_hi=60000,
                                                                     sides=(64, 96, 128, 256))]


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(0x5EED + int(seed))


def _camera_rays(case, seed):
    """Jittered pinhole rays at the mesh from a seeded view direction."""
    W, H = case["width"], case["height"]
    n = W * H
    g = _generator(seed)
    angle = float(torch.rand((), generator=g, device=DEV).item()) * 2 * math.pi
    jitter = torch.rand((n, 2), generator=g, device=DEV) - 0.5
    i = torch.arange(n, device=DEV)
    tan_half = math.tan(math.radians(45.0) / 2)
    x = (((i % W).float() + 0.5 + jitter[:, 0]) / W * 2 - 1) * (tan_half * W / H)
    y = (1 - ((i // W).float() + 0.5 + jitter[:, 1]) / H * 2) * tan_half
    d = torch.stack([x, y, torch.full_like(x, -1.0)], 1)
    d = d / d.norm(dim=1, keepdim=True)
    c, s = math.cos(angle), math.sin(angle)
    turn = torch.tensor([[c, 0, -s], [0, 1, 0], [s, 0, c]], device=DEV)
    rays = torch.zeros((n, 8), device=DEV)
    rays[:, 0:3] = torch.tensor([0.0, 0.0, 3.2], device=DEV) @ turn
    rays[:, 3] = math.inf
    rays[:, 4:7] = d @ turn
    return rays


def _scatter_rays(n, lo, hi, seed, endless=False):
    """Origins uniform in the box, directions uniform on the sphere, tMax
    uniform in [0.1, 2] diagonals (or infinite)."""
    g = _generator(seed)
    lo = torch.as_tensor(np.array(lo, np.float32), device=DEV)
    hi = torch.as_tensor(np.array(hi, np.float32), device=DEV)
    rays = torch.zeros((n, 8), device=DEV)
    rays[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device=DEV)
    d = torch.randn((n, 3), generator=g, device=DEV)
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    diag = float((hi - lo).norm().item())
    rays[:, 3] = math.inf if endless else diag * (0.1 + 1.9 * torch.rand(n, generator=g, device=DEV))
    return rays


def _trace_rays(case, seed):
    if case["rays"] == "camera":
        return _camera_rays(case, seed)
    return _scatter_rays(case["count"], *_sphere(case["subdiv"]).root_bounds(), seed)


def _eye(seed):
    """A seeded view into the box scenes."""
    r = np.random.default_rng(seed)
    return (0.5 + float(r.uniform(-0.1, 0.1)), 0.5 + float(r.uniform(-0.1, 0.1)), 2.2)


def _params(case, seed, width, height, **kw):
    return F.render_params(width, height, case["spp"], max_depth=case["depth"], rr_min_bounce=case.get("rr", case["depth"]),
                           seed=1234 + int(seed), use_graph=1, **kw)


def _films(height, width, count):
    return [torch.zeros((height, width, 3), device=DEV) for _ in range(count)] + [torch.zeros((height, width), device=DEV)]


def _albedo_textures(seed, res):
    """Seeded smooth albedos in [0.1, 0.8]."""
    g = _generator(seed)
    coarse = torch.rand((2, 3, 12, 12), generator=g, device=DEV)
    t = torch.nn.functional.interpolate(coarse, size=(res, res), mode="bilinear", align_corners=True)
    return (0.1 + 0.7 * t).permute(0, 2, 3, 1).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "trace":
        rays = _trace_rays(case, seed)
        n = rays.shape[0]
        st = dict(kind=kind, query=case["query"], acc=GpuAccelerator(_sphere(case["subdiv"])), rays=rays)
        if case["query"] == "closest":
            hits = torch.empty((n, 4), device=DEV)
            st.update(hits=hits, out=dict(t=hits[:, 0], uv=hits[:, 1:3], prim=hits.view(torch.int32)[:, 3]))
        else:
            st.update(prim=torch.empty(n, dtype=torch.int32, device=DEV),
                      occluded=torch.empty(n, dtype=torch.bool, device=DEV))
        return st
    if kind == "host":
        hs = _sphere(case["subdiv"])
        rays = _scatter_rays(case["count"], *hs.root_bounds(), seed).cpu().numpy()
        out = np.zeros(case["count"], F.INTERSECTION_DTYPE)
        return dict(kind=kind, acc=GpuAccelerator(hs), rays=np.ascontiguousarray(rays[:, [0, 1, 2, 4, 5, 6]]),
                    tmax=rays[:, 3].copy(), out=out)
    if kind in ("instances", "field"):
        hosts, inst = _field()
        blas = [GpuAccelerator(h) for h in hosts]
        acc = InstancedAccelerator(blas, inst)
        if kind == "instances":
            rays = _scatter_rays(case["count"], (-24.0,) * 3, (24.0,) * 3, seed, endless=True)
            hits = torch.empty((case["count"], 4), device=DEV)
            which = torch.empty(case["count"], dtype=torch.int32, device=DEV)
            return dict(kind=kind, blas=blas, acc=acc, rays=rays, hits=hits, which=which,
                        out=dict(t=hits[:, 0], uv=hits[:, 1:3], prim=hits.view(torch.int32)[:, 3], instance=which))
        acc.set_environment(_sky(), 1.0)
        acc.set_medium(MEDIUM)
        p = _params(case, seed, case["width"], case["height"], eye=(2.0 * _eye(seed)[0] - 1.0, 6.0, 48.0),
                    target=(0.0, 0.0, 0.0))
        rgb, w = _films(case["height"], case["width"], 1)
        return dict(kind="render", blas=blas, acc=acc, renderer=Renderer(acc, p), films=(rgb, w))
    if kind == "render":
        acc = GpuAccelerator(scenes.box_scene(0xB0 + seed).build())
        p = _params(case, seed, case["width"], case["height"], eye=_eye(seed))
        rgb, w = _films(case["height"], case["width"], 1)
        return dict(kind=kind, acc=acc, renderer=Renderer(acc, p), films=(rgb, w))
    if kind == "materials":
        acc = GpuAccelerator(scenes.materials_box_scene(0xB1 + seed).build())
        p = _params(case, seed, case["width"], case["height"], eye=_eye(seed), mis_corrected=1)
        rgb, sq, alb, nrm, w = _films(case["height"], case["width"], 4)
        return dict(kind=kind, acc=acc, renderer=Renderer(acc, p), films=(rgb, sq, alb, nrm, w))
    if kind == "batch":
        work = _batch(case["scenes"])
        accs = [GpuAccelerator(h) for h, _ in work]
        params = [_params(case, seed + k, side, side, eye=_eye(seed + k)) for k, (_, side) in enumerate(work)]
        br = BatchRenderer(accs, params)
        return dict(kind="render", accs=accs, renderer=br,
                    films=(torch.zeros((br.pixels, 3), device=DEV), torch.zeros(br.pixels, device=DEV)))
    sb, mats = A.adjoint_box_scene(0xB0 + seed)
    acc = GpuAccelerator(sb.build())
    side = case["side"]
    dr = A.DifferentiableRenderer(acc, _params(case, seed, side, side, eye=_eye(seed)), mats)
    g = _generator(seed + 77)
    return dict(kind=kind, acc=acc, dr=dr, texels=_albedo_textures(seed, dr.resolution), scale=0.8,
                target=torch.rand((side, side, 3), generator=g, device=DEV))


def run(st):
    kind = st["kind"]
    if kind == "trace":
        if st["query"] == "closest":
            st["acc"].trace_closest(st["rays"], st["hits"])
            return st["out"]
        st["acc"].trace_any(st["rays"], st["prim"])
        return torch.ge(st["prim"], 0, out=st["occluded"])  # which prim was found first is no answer
    if kind == "host":
        out = st["acc"].intersect_batch(st["rays"], st["tmax"], out=st["out"])
        return dict(t=out["t_hit"], u=out["u"], v=out["v"], hit=out["hit"], id2=out["prim_id"]["id2"])
    if kind == "instances":
        st["acc"].trace_closest(st["rays"], st["hits"], st["which"])
        return st["out"]
    if kind == "render":
        rgb, w = st["films"]
        rgb.zero_()
        w.zero_()
        st["renderer"].render(rgb, w)
        return dict(rgb=rgb, w=w)
    if kind == "materials":
        for f in st["films"]:
            f.zero_()
        rgb, sq, alb, nrm, w = st["films"]
        st["renderer"].render(rgb, w, film_sq=sq, film_albedo=alb, film_normal=nrm)
        return dict(rgb=rgb, sq=sq, albedo=alb, normal=nrm, w=w)
    image, w = st["dr"].forward(st["texels"], st["scale"])
    grad = (image - st["target"]) * (2.0 / image.numel())
    d_tex, d_scale = st["dr"].backward(grad, w, st["texels"], st["scale"])
    return dict(image=image, w=w, d_texels=d_tex, d_scale=d_scale)


# ---------------------------------------------------------------- floors and tolerances


def _ray_count(case):
    return case["width"] * case["height"] if "width" in case else case["count"]


def work(case):
    """Rays in, hits out, geometry once; films out once.  Operations: one
    triangle test a ray (about 50), and for a path vertex the sampling, light
    and BSDF arithmetic that its definition writes out (about 400), with two
    rays; a third of the paths of a roulette render see its last bounce."""
    kind = case["kind"]
    if kind == "trace":
        n = _ray_count(case)
        return dict(bytes=n * (32 + (16 if case["query"] == "closest" else 5)) + 36 * 20 * 4 ** case["subdiv"],
                    flops=50 * n)
    if kind == "host":
        return dict(bytes=case["count"] * (28 + 48), flops=50 * case["count"])
    if kind == "instances":
        return dict(bytes=case["count"] * (32 + 20) + 36 * 16 * 50000 + 96 * 4096, flops=100 * case["count"])
    if kind == "batch":
        pixels = sum(side * side for _, side in _batch(case["scenes"]))
        films, rounds = 16, 1
    elif kind == "adjoint":
        pixels, films, rounds = case["side"] ** 2, 16 + 12, 3  # forward, primal and replay
    else:
        pixels, films, rounds = case["width"] * case["height"], 16 if kind != "materials" else 52, 1
    vertices = pixels * case["spp"] * (1 + 0.6 * (case["depth"] - 1)) * rounds
    return dict(bytes=pixels * films + (2 * 256 * 256 * 12 * 2 if kind == "adjoint" else 0), flops=500 * vertices)


def tolerance(case):
    kind = case["kind"]
    if kind == "trace" and case["query"] == "any":
        return "exact"
    if kind in ("trace", "host", "instances"):
        # 32-bit triangle tests; the nearest of two triangles at the same t is
        # either (about one ray in a million on a shared edge)
        return {"rel": 1e-5, "max": 4e-4, "differ": 1e-5}
    # Film sums in another order are off by about 1e-7.  A change of one unit
    # in the last place somewhere along a path now and then moves it to the
    # other side of an edge or of a roulette decision, and its pixel then holds
    # another, equally valid sample: 32 against 64 bits shows rel 2e-3 in the
    # box scene's image at 16 samples a pixel and 2e-2 in the texel gradients
    # (one path can be most of a texel's gradient).
    if kind == "adjoint":
        return {"rel": 0.03, "max": 0.9, "differ": 1e-5}
    return {"rel": 8e-3, "max": 0.9, "differ": 1e-5}


# ---------------------------------------------------------------- 64 bits: rays against one mesh


def _exact_hits(hs, subdiv, rays):
    """Nearest hit of each ray by descending the icosphere's subdivision
    hierarchy (face i of a level has the children i + k * faces, k = 0..3)
    with box tests, then Moller-Trumbore, all in 64 bits."""
    mesh = hs.meshes[0]
    p = torch.as_tensor(mesh.points[:, :3].astype(np.float64), device=DEV)
    tri = p[torch.as_tensor(mesh.vertex_indices.reshape(-1, 3), device=DEV)]
    lo, hi = tri.amin(1), tri.amax(1)
    levels = [(lo, hi)]
    for _ in range(subdiv):
        lo, hi = lo.view(4, -1, 3).amin(0), hi.view(4, -1, 3).amax(0)
        levels.append((lo, hi))
    levels.reverse()
    n = rays.shape[0]
    t_out = rays[:, 3].double().clone()
    uv_out = torch.zeros((n, 2), dtype=torch.float64, device=DEV)
    for begin in range(0, n, 1 << 18):
        r = rays[begin:begin + (1 << 18)].double()
        o, tmax, d = r[:, 0:3], r[:, 3], r[:, 4:7]
        m = r.shape[0]
        ray = torch.arange(m, device=DEV).repeat_interleave(20)
        face = torch.arange(20, device=DEV).repeat(m)
        for k, (lo, hi) in enumerate(levels):
            a = (lo[face] - o[ray]) / d[ray]
            b = (hi[face] - o[ray]) / d[ray]
            near = torch.minimum(a, b).amax(1).clamp_min(0.0)
            far = torch.minimum(torch.maximum(a, b).amin(1), tmax[ray])
            keep = near <= far * (1 + 1e-9) + 1e-9
            ray, face = ray[keep], face[keep]
            if k < subdiv:
                faces = lo.shape[0]
                ray = ray.repeat_interleave(4)
                face = (face[:, None] + faces * torch.arange(4, device=DEV)).reshape(-1)
        p0, p1, p2 = tri[face].unbind(1)
        t, u, v, ok = _mt(o[ray], d[ray], p0, p1, p2, tmax[ray])
        ray, t, u, v = ray[ok], t[ok], u[ok], v[ok]
        best = torch.full((m,), math.inf, dtype=torch.float64, device=DEV).scatter_reduce(0, ray, t, "amin")
        first = t == best[ray]
        ray, t, u, v = ray[first], t[first], u[first], v[first]
        t_out[begin + ray] = t
        uv_out[begin + ray] = torch.stack([u, v], 1)
    return t_out, uv_out


def _mt(o, d, p0, p1, p2, tmax):
    e1, e2 = p1 - p0, p2 - p0
    pv = torch.linalg.cross(d, e2)
    det = (e1 * pv).sum(-1)
    s = o - p0
    q = torch.linalg.cross(s, e1)
    u = (s * pv).sum(-1) / det
    v = (d * q).sum(-1) / det
    t = (e2 * q).sum(-1) / det
    ok = (det.abs() >= 1e-7) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 0) & (t <= tmax)
    return t, u, v, ok


# ---------------------------------------------------------------- 64 bits: diffuse path tracer

_M32 = 0xFFFFFFFF


def _mix32(x):
    x = x ^ (x >> 16)
    x = (x * 0x85EBCA77) & _M32
    x = x ^ (x >> 13)
    x = (x * 0xC2B2AE35) & _M32
    return x ^ (x >> 16)


def _reverse32(x):
    for shift, mask in ((1, 0x55555555), (2, 0x33333333), (4, 0x0F0F0F0F), (8, 0x00FF00FF)):
        x = ((x & mask) << shift) | ((x >> shift) & mask)
    return ((x << 16) | (x >> 16)) & _M32


def _owen(v, seed):
    v = _reverse32(v)
    v = v ^ ((v * 0x3D20ADEA) & _M32)
    v = (v + seed) & _M32
    v = (v * ((seed >> 16) | 1)) & _M32
    v = v ^ ((v * 0x05526C56) & _M32)
    v = v ^ ((v * 0x53A22864) & _M32)
    return _reverse32(v)


# the 24 permutations of 0..3 of the Z-Sobol index, in the reference's order
_PERMS = ((0, 1, 2, 3), (0, 1, 3, 2), (0, 2, 1, 3), (0, 2, 3, 1), (0, 3, 2, 1), (0, 3, 1, 2), (1, 0, 2, 3), (1, 0, 3, 2),
          (1, 2, 0, 3), (1, 2, 3, 0), (1, 3, 2, 0), (1, 3, 0, 2), (2, 1, 0, 3), (2, 1, 3, 0), (2, 0, 1, 3), (2, 0, 3, 1),
          (2, 3, 0, 1), (2, 3, 1, 0), (3, 1, 2, 0), (3, 1, 0, 2), (3, 2, 1, 0), (3, 2, 0, 1), (3, 0, 2, 1), (3, 0, 1, 2))


class _Sampler:
    """Z-Sobol samples of all paths (Ahmed and Wonka's index permutation over
    Owen-scrambled Sobol points), one running dimension per path."""

    def __init__(self, px, py, sample, width, height, spp, seed):
        morton = torch.zeros_like(px)
        for b in range(16):
            morton |= ((px >> b) & 1) << (2 * b) | ((py >> b) & 1) << (2 * b + 1)
        self.log2spp = spp.bit_length() - 1
        self.morton = (morton << self.log2spp) | sample
        self.dim = torch.zeros_like(px)
        self.seed = seed
        side = 1 << (max(width, height) - 1).bit_length()
        self.digits = side.bit_length() - 1 + (self.log2spp + 1) // 2
        self.perm = torch.tensor(_PERMS, device=DEV)
        self.columns = (torch.quasirandom.SobolEngine(128).sobolstate.to(DEV) << 2) & _M32

    def get(self, count, where):
        """count (1, 2 or 3) numbers of the paths `where`."""
        morton, dim = self.morton[where], self.dim[where]
        product = 0x55555555 * dim
        fold = (product & _M32) ^ (product >> 32)

        def mixed(higher):
            return _mix32((higher & _M32) ^ (higher >> 32) ^ fold)

        odd = self.log2spp & 1
        index = torch.zeros_like(morton)
        for i in range(self.digits - 1, odd - 1, -1):
            shift = 2 * i - odd
            digit = (morton >> shift) & 3
            index |= self.perm[(mixed(morton >> (shift + 2)) >> 24) % 24, digit] << shift
        if odd:
            index |= (morton & 1) ^ (mixed(morton >> 1) & 1)
        out = []
        for k in range(count):
            bits = torch.zeros_like(index)
            for b in range(30):
                bits ^= torch.where((index >> b) & 1 != 0, self.columns[dim + k, b], 0)
            key = dim + k
            scramble = torch.zeros_like(dim) if k == 1 else _mix32(((key ^ self.seed) & _M32) ^ ((key ^ self.seed) >> 32))
            out.append((_owen(bits, scramble).double() * 2.0 ** -32).clamp_max(1 - 1e-6))
        self.dim[where] += count
        return out


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _dot(a, b):
    return (a * b).sum(-1)


def _axes(n):
    """A coordinate system around n."""
    x, y, z = n.unbind(-1)
    zero = torch.zeros_like(x)
    a = torch.stack([-z, zero, x], -1) / (x * x + z * z).sqrt()[:, None]
    b = torch.stack([zero, z, -y], -1) / (y * y + z * z).sqrt()[:, None]
    v2 = torch.where((x.abs() > y.abs())[:, None], a, b)
    return v2, torch.linalg.cross(n, v2)


def _cosine(u0, u1):
    ox, oy = 2 * u0 - 1, 2 * u1 - 1
    wide = ox.abs() > oy.abs()
    r = torch.where(wide, ox, oy)
    theta = torch.where(wide, math.pi / 4 * (oy / ox), math.pi / 2 - math.pi / 4 * (ox / oy))
    x, y = r * theta.cos(), r * theta.sin()
    return torch.stack([x, y, (1 - x * x - y * y).clamp_min(0).sqrt()], -1)


def _gauss(u, radius, sigma):
    norm = 0.5 * (1 + math.erf(radius / (sigma * math.sqrt(2))))
    x = sigma * math.sqrt(2) * torch.erfinv(2 * ((1 - norm) + u * (2 * norm - 1)) - 1)
    pdf = torch.exp(-x * x / (2 * sigma * sigma)) / (sigma * math.sqrt(2 * math.pi)) / (2 * norm - 1)
    x = x.clamp(-radius, radius)
    value = torch.exp(-x * x / (2 * sigma * sigma)) / math.sqrt(2 * math.pi * sigma * sigma)
    return x, value / pdf


class _Boxes:
    """The triangles, materials and lights of a small diffuse host scene, in 64
    bits; rays are tested against every triangle."""

    def __init__(self, hs):
        prims = hs.prims
        which = prims["id2"].astype(np.int64)
        mesh, tri = which >> 32, which & 0xFFFFFFFF
        corners = np.stack([hs.meshes[m].points[hs.meshes[m].vertex_indices.reshape(-1, 3)[t], :3] for m, t in zip(mesh, tri)])
        self.p = torch.as_tensor(corners.astype(np.float64), device=DEV)
        self.material = torch.as_tensor(prims["material_index"].astype(np.int64), device=DEV)
        self.is_light = torch.as_tensor(prims["type"] == 3, device=DEV)
        self.albedo = torch.as_tensor(np.array(hs.materials["albedo"], np.float64), device=DEV)
        self.emission = torch.as_tensor(np.array(hs.materials["emission"], np.float64), device=DEV)
        lights = np.nonzero(prims["type"] == 3)[0]
        self.lights = torch.as_tensor(lights[np.argsort(prims["id1"][lights], kind="stable")], device=DEV)
        p0, p1, p2 = self.p[self.lights].unbind(1)
        self.area = 0.5 * torch.linalg.cross(p1 - p0, p2 - p0).norm(dim=1)
        self.power = self.emission[self.material[self.lights]].mean(1) * self.area * math.pi

    def nearest(self, o, d, tmax):
        best = torch.full((o.shape[0],), float(tmax), dtype=torch.float64, device=DEV)
        prim = torch.full((o.shape[0],), -1, device=DEV)
        u = torch.zeros_like(best)
        v = torch.zeros_like(best)
        for k in range(self.p.shape[0]):
            p0, p1, p2 = (x.expand_as(o) for x in self.p[k])
            tk, uk, vk, ok = _mt(o, d, p0, p1, p2, best)
            best, u, v = torch.where(ok, tk, best), torch.where(ok, uk, u), torch.where(ok, vk, v)
            prim = torch.where(ok, k, prim)
        return prim, u, v


def _exact_paths(hs, p, albedo_of, scale=1.0):
    """Radiance (with autograd through albedo_of and scale), film weight and
    pixel of every path of the frame: the integrator with MIS as written (the
    BSDF strategy weighs nothing), diffuse surfaces, area lights."""
    box = _Boxes(hs)
    W, H, spp = p.width, p.height, p.spp
    path = torch.arange(W * H * spp, device=DEV)
    pixel = path // spp
    px, py = pixel % W, pixel // W
    z = _Sampler(px, py, path % spp, W, H, spp, p.seed)
    every = torch.ones_like(path, dtype=torch.bool)
    u0, u1 = z.get(2, every)
    dx, wx = _gauss(u0, p.filter_radius, p.filter_sigma)
    dy, wy = _gauss(u1, p.filter_radius, p.filter_sigma)
    z.get(2, every)  # lens
    tan_half = math.tan(math.radians(p.fov_deg) / 2)
    aspect = W / H
    sx, sy = (aspect, 1.0) if aspect > 1 else (1.0, 1.0 / aspect)
    cam = torch.stack([(-sx + (px + 0.5 + dx) / W * 2 * sx) * tan_half, (sy - (py + 0.5 + dy) / H * 2 * sy) * tan_half,
                       torch.ones_like(dx)], -1)
    cam = _unit(cam)
    eye, target, up = (torch.tensor(list(v), dtype=torch.float64, device=DEV) for v in (p.eye, p.target, p.up))
    fwd = _unit(target - eye)
    right = _unit(torch.linalg.cross(fwd, up))
    d = cam[:, 0:1] * right + cam[:, 1:2] * torch.linalg.cross(right, fwd) + cam[:, 2:3] * fwd
    o = eye.expand_as(d)
    L = torch.zeros_like(d)
    thr = torch.ones_like(d)
    live = path
    total = box.power.sum()
    cdf = box.power.cumsum(0)
    for bounce in range(p.max_depth):
        prim, u, v = box.nearest(o, d, math.inf)
        hit = prim >= 0
        live, o, d, thr, prim, u, v = (x[hit] for x in (live, o, d, thr, prim, u, v))
        p0, p1, p2 = box.p[prim].unbind(1)
        pos = p0 * (1 - u - v)[:, None] + p1 * u[:, None] + p2 * v[:, None]
        n = _unit(torch.linalg.cross(p0 - p2, p1 - p2))
        wo = -_unit(d)
        light = box.is_light[prim]
        if bounce == 0:
            le = torch.where((light & (_dot(n, wo) > 0))[:, None], box.emission[box.material[prim]] * scale, 0.0)
            L = L.index_add(0, live, thr * le)
        refl = albedo_of(torch.where(light, 0, box.material[prim]), pos)
        f = refl / math.pi
        # the shading frame
        s = _unit(_axes(_unit(torch.linalg.cross(p2 - p0, p1 - p0)))[0])
        t = _unit(torch.linalg.cross(s, n))
        fy = _unit(torch.linalg.cross(t, n))
        fx = torch.linalg.cross(fy, n)
        wo_z = _dot(wo, n)
        # one light sample
        (uc,) = z.get(1, live)
        which = torch.searchsorted(cdf, uc * total).clamp_max(len(cdf) - 1)
        choose = box.power[which] / total
        u0, u1 = z.get(2, live)
        l0, l1, l2 = box.p[box.lights[which]].unbind(1)
        su0 = u0.sqrt()
        b0, b1 = (1 - su0)[:, None], (u1 * su0)[:, None]
        on_light = l0 * b0 + l1 * b1 + l2 * ((1 - b0) - b1)
        ln = _unit(torch.linalg.cross(l1 - l0, l2 - l0))
        inc = _unit(on_light - pos)
        facing = -_dot(ln, inc)
        pdf = (1 / box.area[which]) * ((pos - on_light) ** 2).sum(-1) / facing.abs()
        same_side = _dot(inc, n) * wo_z > 0
        bsdf_pdf = torch.where(same_side & (wo_z != 0), _dot(inc, n).abs() / math.pi, 0.0)
        weight = torch.where(bsdf_pdf > 0, pdf * pdf / (pdf * pdf + bsdf_pdf * bsdf_pdf), 0.0)
        use = (facing > 0) & torch.isfinite(pdf) & same_side
        start = pos + (on_light - pos) * 0.0001
        blocked = box.nearest(start, on_light - start, 1 - 0.00001)[0] >= 0
        gain = torch.where(use & ~blocked, _dot(inc, n).abs() * weight / pdf / choose, 0.0)
        L = L.index_add(0, live, thr * f * (box.emission[box.material[box.lights[which]]] * scale) * gain[:, None])
        z.get(3, live)  # the BSDF strategy's numbers
        v0, v1, _ = z.get(3, live)
        wi = _cosine(v0, v1)
        wi = torch.where((wo_z < 0)[:, None], wi * torch.tensor([1.0, 1.0, -1.0], device=DEV, dtype=torch.float64), wi)
        pdf_c = torch.where(wo_z * wi[:, 2] > 0, wi[:, 2].abs() / math.pi, 0.0)
        world = fx * wi[:, 0:1] + fy * wi[:, 1:2] + n * wi[:, 2:3]
        go = pdf_c > 0
        thr = thr * f * (_dot(world, n).abs() / torch.where(go, pdf_c, 1.0))[:, None]
        side = torch.where((_dot(world, n) > 0)[:, None], n, -n)
        o = pos + side * 0.0001
        with torch.no_grad():
            most = thr.amax(-1)
            roulette = go & (most < 1) & (bounce >= p.rr_min_bounce)
            if bool(roulette.any()):
                stop = (1 - most).clamp_min(0)
                (ur,) = z.get(1, live[roulette])
                go[roulette] &= ur >= stop[roulette]
        if bounce >= p.rr_min_bounce:
            thr = torch.where(roulette[:, None], thr / torch.where(roulette, most, 1.0)[:, None], thr)
        live, o, d, thr = live[go], o[go], world[go], thr[go]
    return L, wx * wy, pixel


def _film(L, w, pixel, width, height):
    rgb = torch.zeros((width * height, 3), dtype=torch.float64, device=DEV).index_add(0, pixel, L)
    return rgb.view(height, width, 3), torch.zeros(width * height, dtype=torch.float64, device=DEV).index_add(
        0, pixel, w).view(height, width)


def exact(case, seed):
    kind = case["kind"]
    if kind == "trace" and case["query"] == "closest":
        t, uv = _exact_hits(_sphere(case["subdiv"]), case["subdiv"], _trace_rays(case, seed))
        return dict(t=t, uv=uv, prim=None)
    if kind == "host":
        hs = _sphere(case["subdiv"])
        t, uv = _exact_hits(hs, case["subdiv"], _scatter_rays(case["count"], *hs.root_bounds(), seed))
        return dict(t=t, u=uv[:, 0].contiguous(), v=uv[:, 1].contiguous(), hit=None, id2=None)
    if kind == "render":
        hs = scenes.box_scene(0xB0 + seed).build()
        p = _params(case, seed, case["width"], case["height"], eye=_eye(seed))
        albedo = _Boxes(hs).albedo
        rgb, w = _film(*_exact_paths(hs, p, lambda m, pos: albedo[m]), case["width"], case["height"])
        return dict(rgb=rgb, w=w)
    if kind == "adjoint":
        sb, mats = A.adjoint_box_scene(0xB0 + seed)
        hs = sb.build()
        side, res = case["side"], A.TEXTURE_RES
        p = _params(case, seed, side, side, eye=_eye(seed))
        albedo = _Boxes(hs).albedo
        texels = _albedo_textures(seed, res).double().requires_grad_()
        scale = torch.tensor(float(np.float32(0.8)), dtype=torch.float64, device=DEV, requires_grad=True)

        def albedo_of(m, pos):
            refl = albedo[m]
            for k, (material, (org, ua, va)) in enumerate(zip(mats, (A.FLOOR, A.BACK_WALL))):
                q = pos - torch.tensor(org, dtype=torch.float64, device=DEV)
                ix, iy = ((_dot(q, torch.tensor(a, dtype=torch.float64, device=DEV)) * res).clamp(0, res - 1).long()
                          for a in (ua, va))
                refl = torch.where((m == material)[:, None], texels[k][iy, ix], refl)
            return refl

        rgb, w = _film(*_exact_paths(hs, p, albedo_of, scale), side, side)
        image = rgb / w[..., None]
        g = _generator(seed + 77)
        target = torch.rand((side, side, 3), generator=g, device=DEV)
        d_tex, d_scale = torch.autograd.grad(image, [texels, scale], (image.detach() - target) * (2.0 / image.numel()))
        return dict(image=image.detach(), w=w, d_texels=d_tex, d_scale=d_scale)
    # any hit is yes or no; 4096 instances of 50,000 triangles, random walks in
    # layers and eight scenes' trees take minutes in plain torch
    return None
