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
