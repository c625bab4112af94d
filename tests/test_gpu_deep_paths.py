"""Queue counters of many bounces: a renderer keeps one block of them per bounce
of its deepest scene.  Roulette ends every path long before the depth, so a far
larger depth renders the same image from the same rays."""
import numpy as np
import pytest

from gonzales_b200 import GpuAccelerator, scenes
from gonzales_b200 import _ffi as F

pytestmark = pytest.mark.gpu

RAYS = ["camera_rays", "extension_rays", "shadow_rays", "probe_rays"]


@pytest.mark.parametrize("graph", [0, 1])
def test_depth_beyond_every_path_changes_nothing(graph):
    with GpuAccelerator(scenes.box_scene().build()) as acc:
        base = dict(width=32, height=24, spp=4, rr_min_bounce=2, mis_corrected=1, use_graph=graph)
        a = acc.render(F.render_params(max_depth=150, **base))
        b = acc.render(F.render_params(max_depth=1200, **base))
        assert [a[3][k] for k in RAYS] == [b[3][k] for k in RAYS]
        for x, y in zip(a[:3], b[:3]):
            np.testing.assert_allclose(x, y, rtol=1e-5, atol=1e-6)  # the order of the film's atomics
        assert acc.error_word() == 0
