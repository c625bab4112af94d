"""The traversal kernels with a warp's triangle queue against those that test
lane by lane.  A launch of more than 400 rays per wide node takes the latter, so
the same rays traced in small slices and all at once go through both: hits must
be bit-identical: closest hits with both leaf tests, and the first prim that any
hit finds.  Scenes: nodes whose leaves hold more triangles than a queue takes from a
lane at once, equal-t ties (coincident triangles), tiny trees, two levels; slices
that do not fill a warp."""
import numpy as np
import pytest

from gonzales_b200 import GpuAccelerator, InstancedAccelerator, options, scenes
from gonzales_b200 import _ffi as F
from tests.test_gpu_traversal import _edge_scene

pytestmark = pytest.mark.gpu


def _coincident(rng):
    """Stacks of identical triangles: every hit is an equal-t tie."""
    sb = scenes.SceneBuilder()
    m = sb.add_material()
    for _ in range(30):
        pts = rng.uniform(-1, 1, (3, 3)).astype(np.float32)
        for _ in range(5):
            sb.add_mesh(pts, [[0, 1, 2]], m)
    return sb.build()


def _rays(rng, n, scale=1.0):
    dirs = rng.normal(size=(n, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    o = dirs * 4.0 * scale
    d = rng.normal(scale=0.5 * scale, size=(n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    t = np.where(rng.random(n) < 0.3, rng.uniform(2, 6, n) * scale, np.inf)
    return scenes.pack_device_rays(o.astype(np.float32), d.astype(np.float32), t.astype(np.float32))


def _slices(n, step):
    return [slice(k, min(k + step, n)) for k in range(0, n, step)]


SCENES = ["1", "3", "9", "same-centroid", "grid", "coincident"]


@pytest.mark.parametrize("kind", SCENES)
@pytest.mark.parametrize("leaf", [F.LEAF_MOLLER_TRUMBORE, F.LEAF_WATERTIGHT])
def test_queue_equals_lane_tests(kind, leaf):
    import torch

    rng = np.random.default_rng(len(kind) + 100 * leaf)
    hs = _coincident(rng) if kind == "coincident" else _edge_scene(kind, rng)
    with GpuAccelerator(hs) as acc:
        nodes = acc.info()["wide_nodes"]
        n = 400 * nodes + 777
        rays = torch.from_numpy(_rays(rng, n)).cuda()
        opt = options(leaf_test=leaf)
        whole = torch.empty((n, 4), device="cuda")
        acc.trace_closest(rays, whole, opt)
        any_whole = torch.empty(n, dtype=torch.int32, device="cuda")
        acc.trace_any(rays, any_whole, opt)
        for step in (1 + 400 * nodes // 3, 333):
            got = torch.empty((n, 4), device="cuda")
            any_got = torch.empty(n, dtype=torch.int32, device="cuda")
            for s in _slices(n, min(step, 400 * nodes))[:40]:
                acc.trace_closest(rays[s], got[s], opt)
                acc.trace_any(rays[s], any_got[s], opt)
            m = min(n, 40 * min(step, 400 * nodes))
            torch.cuda.synchronize()
            assert got[:m].cpu().numpy().tobytes() == whole[:m].cpu().numpy().tobytes()
            assert torch.equal(any_got[:m], any_whole[:m])
        hit = whole[:, 3].view(torch.int32) >= 0
        assert bool(hit.any()) and torch.equal(hit, any_whole >= 0)
        assert acc.error_word() == 0


@pytest.mark.parametrize("n_instances", [1, 7, 60])
def test_two_level_queue_equals_lane_tests(n_instances):
    import torch

    rng = np.random.default_rng(n_instances)
    hosts, _ = scenes.instanced_scene(n_meshes=2, n_u=5, n_v=4, n_instances=1)
    inst = scenes.random_instances(n_instances, 2, 5, extent=1.5)
    blas = [GpuAccelerator(h) for h in hosts]
    with InstancedAccelerator(blas, inst) as acc:
        nodes = acc.info()["wide_nodes"]
        n = 400 * nodes + 555
        rays = torch.from_numpy(_rays(rng, n, 1.5)).cuda()
        whole, w_inst = torch.empty((n, 4), device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        acc.trace_closest(rays, whole, w_inst)
        any_whole = torch.empty(n, dtype=torch.int32, device="cuda")
        acc.trace_any(rays, any_whole)
        got, g_inst = torch.empty_like(whole), torch.empty_like(w_inst)
        any_got = torch.empty_like(any_whole)
        for s in _slices(n, 1 + n // 7):
            acc.trace_closest(rays[s], got[s], g_inst[s])
            acc.trace_any(rays[s], any_got[s])
        torch.cuda.synchronize()
        assert got.cpu().numpy().tobytes() == whole.cpu().numpy().tobytes()
        assert torch.equal(g_inst, w_inst) and bool((w_inst >= 0).any())
        assert torch.equal(any_got, any_whole)
        assert acc.error_word() == 0
    for b in blas:
        b.close()


def _both_ways(acc, rays, n, opt, step):
    """Closest hits and first prims of one launch (lane tests) and of slices (queue)."""
    import torch

    hits = [torch.empty((n, 4), device="cuda") for _ in range(2)]
    prim = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]
    acc.trace_closest(rays, hits[0], opt)
    acc.trace_any(rays, prim[0], opt)
    for s in _slices(n, step):
        acc.trace_closest(rays[s], hits[1][s], opt)
        acc.trace_any(rays[s], prim[1][s], opt)
    torch.cuda.synchronize()
    return [h.cpu().numpy() for h in hits], [p.cpu().numpy() for p in prim]


@pytest.mark.parametrize("kind", ["9", "grid"])
@pytest.mark.parametrize("leaf", [F.LEAF_MOLLER_TRUMBORE, F.LEAF_WATERTIGHT])
def test_a_nan_limit_gives_one_answer(kind, leaf):
    """A ray whose tMax is NaN is limited by nothing in the leaf tests; the
    queue, the lane tests and the one-ray-per-thread kernel say the same."""
    import torch

    rng = np.random.default_rng(7)
    with GpuAccelerator(_edge_scene(kind, rng)) as acc:
        nodes = acc.info()["wide_nodes"]
        n = 400 * nodes + 777
        host = _rays(rng, n)
        host[::3, 3] = np.nan
        rays = torch.from_numpy(host).cuda()
        hits, prim = _both_ways(acc, rays, n, options(leaf_test=leaf), 1 + 130 * nodes)
        assert hits[0].tobytes() == hits[1].tobytes()
        assert np.array_equal(prim[0], prim[1])
        one = torch.empty((n, 4), device="cuda")
        acc.trace_closest(rays, one, options(leaf_test=leaf, traversal=F.TRAVERSAL_WIDE_ONE_RAY_PER_THREAD))
        torch.cuda.synchronize()
        assert one.cpu().numpy().tobytes() == hits[0].tobytes()
        nan = np.isnan(host[:, 3])
        assert (hits[0][nan, 3].view(np.int32) >= 0).any()


def test_two_level_nan_limit_gives_one_answer():
    import torch

    rng = np.random.default_rng(8)
    hosts, _ = scenes.instanced_scene(n_meshes=2, n_u=5, n_v=4, n_instances=1)
    blas = [GpuAccelerator(h) for h in hosts]
    with InstancedAccelerator(blas, scenes.random_instances(7, 2, 5, extent=1.5)) as acc:
        n = 400 * acc.info()["wide_nodes"] + 555
        host = _rays(rng, n, 1.5)
        host[::3, 3] = np.nan
        rays = torch.from_numpy(host).cuda()
        hits = [torch.empty((n, 4), device="cuda") for _ in range(2)]
        inst = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]
        acc.trace_closest(rays, hits[0], inst[0])
        for s in _slices(n, 1 + n // 5):
            acc.trace_closest(rays[s], hits[1][s], inst[1][s])
        torch.cuda.synchronize()
        assert hits[0].cpu().numpy().tobytes() == hits[1].cpu().numpy().tobytes()
        assert torch.equal(inst[0], inst[1]) and bool((inst[0][::3] >= 0).any())
    for b in blas:
        b.close()


def _slivers(rng, count):
    """Needles in the plane y = 0, on top of one another: a ray meets several
    at the same distance, which their tests compute with relative errors of
    1e-7 to 1e-4, well past a box's slack."""
    sb = scenes.SceneBuilder()
    m = sb.add_material()
    c, a = rng.uniform(0, 1, (count, 2)), rng.uniform(0, 2 * np.pi, count)
    along = 0.5 * np.stack([np.cos(a), np.sin(a)], 1)
    across = rng.uniform(2e-4, 2e-2, (count, 1)) * np.stack([-np.sin(a), np.cos(a)], 1)
    p = np.stack([c - along, c + along, c + across], 1).reshape(-1, 2)
    pts = np.stack([p[:, 0], np.zeros(len(p)), p[:, 1]], 1).astype(np.float32)
    sb.add_mesh(pts, np.arange(3 * count).reshape(-1, 3), m)
    return sb.build()


def _grazing_rays(rng, n):
    target = np.stack([rng.uniform(0, 1, n), np.zeros(n), rng.uniform(0, 1, n)], 1)
    a, e = rng.uniform(0, 2 * np.pi, n), 10.0 ** rng.uniform(-2, 0, n)
    d = np.stack([np.cos(a), -e, np.sin(a)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = target - d * 10.0 ** rng.uniform(0, 1.5, (n, 1))
    rays = scenes.pack_device_rays(o.astype(np.float32), d.astype(np.float32), np.full(n, np.inf, np.float32))
    rays[::1000, 5] = np.nan  # a direction with a NaN: every distance is one
    return rays


@pytest.mark.parametrize("leaf", [F.LEAF_MOLLER_TRUMBORE, F.LEAF_WATERTIGHT])
def test_a_rays_hit_depends_on_the_ray_alone(leaf):
    """Triangles whose computed distance falls before their own box: which
    nodes a ray has opened before its queued triangles are tested must not
    decide its hit.  The one-ray-per-thread kernel prunes at once."""
    import torch

    rng = np.random.default_rng(21)
    with GpuAccelerator(_slivers(rng, 4000)) as acc:
        n = 390 * acc.info()["wide_nodes"]
        rays = torch.from_numpy(_grazing_rays(rng, n)).cuda()
        order = torch.from_numpy(rng.permutation(n)).cuda()
        one, got, mixed = (torch.empty((n, 4), device="cuda") for _ in range(3))
        acc.trace_closest(rays, one, options(leaf_test=leaf, traversal=F.TRAVERSAL_WIDE_ONE_RAY_PER_THREAD))
        acc.trace_closest(rays, got, options(leaf_test=leaf))
        acc.trace_closest(rays[order].contiguous(), mixed, options(leaf_test=leaf))
        torch.cuda.synchronize()
        bits = one.view(torch.int32)
        assert int((got.view(torch.int32) != bits).any(1).sum()) == 0
        assert int((mixed.view(torch.int32) != bits[order]).any(1).sum()) == 0
        assert bool((bits[:, 3] >= 0).any()) and acc.error_word() == 0


def test_two_level_hit_depends_on_the_ray_alone():
    import torch

    rng = np.random.default_rng(22)
    blas = [GpuAccelerator(_slivers(rng, 1000)) for _ in range(2)]
    with InstancedAccelerator(blas, scenes.random_instances(6, 2, 5, extent=0.3)) as acc:
        n = 400 * acc.info()["wide_nodes"] + 555
        rays = torch.from_numpy(_grazing_rays(rng, n)).cuda()
        whole, w_inst = torch.empty((n, 4), device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        got, g_inst = torch.empty_like(whole), torch.empty_like(w_inst)
        acc.trace_closest(rays, whole, w_inst)
        for s in _slices(n, 1 + n // 5):
            acc.trace_closest(rays[s], got[s], g_inst[s])
        torch.cuda.synchronize()
        bad = (got.view(torch.int32) != whole.view(torch.int32)).any(1) | (g_inst != w_inst)
        assert int(bad.sum()) == 0
        assert bool((w_inst >= 0).any()) and acc.error_word() == 0
    for b in blas:
        b.close()


@pytest.mark.parametrize("leaf", [F.LEAF_MOLLER_TRUMBORE, F.LEAF_WATERTIGHT])
def test_dense_sphere_hits_depend_on_the_ray_alone(leaf):
    """Rays at the vertices and edges of a dense sphere and along its surface."""
    import torch

    pts, tris = scenes.displaced_icosphere(7, seed=3)
    sb = scenes.SceneBuilder()
    sb.add_mesh(pts, tris, sb.add_material())
    rng = np.random.default_rng(23)
    n = 2_000_000
    pick = tris[rng.integers(0, len(tris), n)]
    s = rng.uniform(0, 1, (n, 1)) * (rng.random((n, 1)) < 0.7)  # the rest at a vertex
    target = (1 - s) * pts[pick[:, 0]] + s * pts[pick[:, 1]]
    out = target / np.linalg.norm(target, axis=1, keepdims=True)
    d = rng.normal(size=(n, 3))
    d -= out * (d * out).sum(1, keepdims=True) * rng.choice([0.0, 0.97, 1.0], (n, 1))  # a third tangent, a third nearly
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (target - 3.0 * d).astype(np.float32)
    with GpuAccelerator(sb.build()) as acc:
        rays = torch.from_numpy(scenes.pack_device_rays(o, d.astype(np.float32), np.full(n, np.inf, np.float32))).cuda()
        one, got = torch.empty((n, 4), device="cuda"), torch.empty((n, 4), device="cuda")
        acc.trace_closest(rays, one, options(leaf_test=leaf, traversal=F.TRAVERSAL_WIDE_ONE_RAY_PER_THREAD))
        acc.trace_closest(rays, got, options(leaf_test=leaf))
        torch.cuda.synchronize()
        assert int((got.view(torch.int32) != one.view(torch.int32)).any(1).sum()) == 0
        assert bool((one[:, 3].view(torch.int32) >= 0).any())


@pytest.mark.parametrize("depth", [8, 16, 32, 64])
def test_requested_stack_depth_does_not_choose_the_kernel(depth):
    """A launch of more than 400 rays a node tests lane by lane whatever stack
    the caller asks for: node and triangle fetches are those of the kernel that
    prunes at once (the queue adds some), hits and any hits the same."""
    import torch

    with GpuAccelerator(_edge_scene("grid", np.random.default_rng(3))) as acc:
        n = 400 * acc.info()["wide_nodes"] + 777
        rays = torch.from_numpy(_rays(np.random.default_rng(4), n)).cuda()
        got = []
        for o in (dict(traversal=F.TRAVERSAL_WIDE_ONE_RAY_PER_THREAD), dict(stack_depth=depth)):
            count = torch.zeros(3, dtype=torch.int64, device="cuda")
            hits = torch.empty((n, 4), device="cuda")
            acc.trace_closest(rays, hits, options(fetch_counters=count.data_ptr(), **o))
            torch.cuda.synchronize()
            got.append((hits.cpu().numpy().tobytes(), count.cpu().tolist()))
        assert got[0] == got[1]
        assert acc.error_word() == 0
