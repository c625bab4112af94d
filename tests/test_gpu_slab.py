"""The wide nodes' slab test where its folded constants round most: scenes far
from the origin, rays from far away, directions with zero and tiny components,
and a tree so large that the reciprocal directions are bounded below 2^64.  A
box may be entered too often, never missed: every ray's closest hit is the
oracle's exactly (or a counted tie or reference-culled hit), on trees converted
on the host and built on the device."""
import numpy as np
import pytest

from gonzales_b200 import GpuAccelerator, scenes
from tests import helpers as H
from tests.test_gpu_traversal import _check, device_any, device_closest

pytestmark = pytest.mark.gpu


def _scene(kind, scale, offset):
    sb = scenes.SceneBuilder()
    m = sb.add_material()
    pts, tris = scenes.displaced_icosphere(3, seed=11)
    sb.add_mesh((pts * np.float32(scale) + np.asarray(offset, np.float32)).astype(np.float32), tris, m)
    if kind == "huge":  # one triangle far larger than all else
        big = np.array([[-1, -1e17, -1e17], [-1, 2e17, -1e17], [-1, -1e17, 2e17]], np.float32) - np.float32(4 * scale)
        sb.add_mesh(big, [[0, 1, 2]], m)
    return sb.build()


def _rays(rng, scale, offset, far, n=6000):
    """Rays through the mesh's neighbourhood from `far` extents away; a third
    along an axis, a third with tiny off-axis components."""
    d = rng.normal(size=(n, 3))
    axis = rng.integers(0, 3, n)
    sign = rng.choice([-1.0, 1.0], n)
    for k in range(n):
        if k % 3 < 2:
            d[k] = 0.0 if k % 3 == 0 else d[k] * 10.0 ** -rng.integers(4, 24)
            d[k, axis[k]] = sign[k]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    aim = rng.uniform(-1.1, 1.1, (n, 3)) * scale
    aim[::10] = np.round(aim[::10] * 4) / 4  # on grid lines
    o = aim + np.asarray(offset) - d * far * scale
    return o.astype(np.float32), d.astype(np.float32), np.full(n, np.inf, np.float32)


CASES = [("plain", 1.0, (0, 0, 0), 3.0), ("plain", 1.0, (0, 0, 0), 3000.0), ("plain", 0.125, (900.0, -700.0, 20.0), 2.0),
         ("plain", 2.0 ** 9, (0, 0, 0), 0.5), ("plain", 2.0 ** 9, (3e4, 0, -3e4), 40.0), ("huge", 1.0, (0, 0, 0), 3.0)]


@pytest.mark.parametrize("kind,scale,offset,far", CASES)
@pytest.mark.parametrize("device_build", [False, True])
def test_slab_is_conservative(kind, scale, offset, far, device_build):
    hs = _scene(kind, scale, offset)
    o, d, t = _rays(np.random.default_rng(int(far * 10) + device_build), scale, offset, far)
    isect, idx, _ = H.oracle_closest(hs, o, d, t)
    assert (idx >= 0).any()
    with GpuAccelerator(hs, device_build=device_build) as acc:
        gpu = device_closest(acc, o, d, t)
        counts, fails = _check(hs, o, d, t, gpu, isect, idx)
        assert counts["fail"] == 0, (counts, fails[:5])
        hit = device_any(acc, o, d, t) >= 0
        assert np.all(hit[idx >= 0])
        assert acc.error_word() == 0
