"""Film sums of a pass: warps add the samples of a pixel together before the
atomics, AOV state is kept only when an AOV film is asked for, and queue counters
are kept per bounce.  The float films must equal the double-precision films of
the same paths (added one by one) to the rounding of at most spp float
additions, at sample counts that do and do not divide a warp, for waves that
split a pixel's samples and for batches of scenes."""
import numpy as np
import pytest

from gonzales_b200 import BatchRenderer, GpuAccelerator, Renderer, scenes
from gonzales_b200 import _ffi as F

pytestmark = pytest.mark.gpu


def _films(n, dtype):
    import torch

    return torch.zeros((n, 3), dtype=dtype, device="cuda"), torch.zeros((n, 3), dtype=dtype, device="cuda"), \
        torch.zeros(n, dtype=dtype, device="cuda")


def _compare(renderer, pixels, spp):
    import torch

    rgb, sq, w = _films(pixels, torch.float32)
    drgb, dsq, dw = _films(pixels, torch.float64)
    renderer.render(rgb, w, film_sq=sq)
    F.check(F.lib().gzg_renderer_render_f64(renderer.handle, drgb.data_ptr(), dsq.data_ptr(), dw.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    # every term is non-negative: a float sum of n terms in any order is within
    # n 2^-24 of the exact one, and a squared term carries one more rounding
    for a, b in ((rgb, drgb), (sq, dsq), (w, dw)):
        a, b = a.cpu().numpy().astype(np.float64), b.cpu().numpy()
        assert b.max() > 0
        assert np.all(np.abs(a - b) <= (spp + 1) * 2.0 ** -24 * b + 1e-30)


@pytest.mark.parametrize("spp", [1, 2, 3, 5, 16, 31, 32, 33, 40])
@pytest.mark.parametrize("wave_paths", [0, 1001])
def test_float_films_equal_double_films(spp, wave_paths):
    with GpuAccelerator(scenes.box_scene().build()) as acc:
        p = F.render_params(23, 17, spp, max_depth=4, rr_min_bounce=2, wave_paths=wave_paths)
        with Renderer(acc, p) as r:
            _compare(r, 23 * 17, spp)
            rays = r.stats()
            assert rays["camera_rays"] == 2 * 23 * 17 * spp
            assert rays["extension_rays"] > rays["camera_rays"] and rays["shadow_rays"] > 0


def test_batch_films_equal_double_films():
    accs = [GpuAccelerator(scenes.box_scene(k).build()) for k in (1, 2, 3)]
    params = [F.render_params(s, s + 1, spp, max_depth=d, rr_min_bounce=2) for s, spp, d in ((9, 7, 2), (16, 12, 5), (5, 3, 1))]
    with BatchRenderer(accs, params, wave_paths=700) as br:
        _compare(br, br.pixels, 12)
    for a in accs:
        a.close()


@pytest.mark.parametrize("which", ["albedo", "normal", "both"])
def test_aov_films_one_at_a_time(which):
    """Passes with one AOV film, both or none on one renderer: each film is the
    one of a pass with both."""
    import torch

    with GpuAccelerator(scenes.materials_box_scene().build()) as acc:
        p = F.render_params(31, 19, 6, max_depth=3, rr_min_bounce=2, use_graph=1)
        with Renderer(acc, p) as r:
            def run(albedo, normal):
                out = [torch.zeros((31 * 19, 3), device="cuda") for _ in range(3)] + [torch.zeros(31 * 19, device="cuda")]
                r.render(out[0], out[3], film_albedo=out[1] if albedo else None, film_normal=out[2] if normal else None)
                torch.cuda.synchronize()
                return [x.cpu().numpy() for x in out]

            plain = run(False, False)
            both = run(True, True)
            one = run(which != "normal", which != "albedo")
            np.testing.assert_allclose(plain[0], both[0], rtol=6 * 2.0 ** -23)
            np.testing.assert_allclose(one[0], both[0], rtol=6 * 2.0 ** -23)
            if which != "normal":
                np.testing.assert_allclose(one[1], both[1], rtol=6 * 2.0 ** -23)
                assert both[1].max() > 0
            if which != "albedo":
                np.testing.assert_allclose(one[2], both[2], rtol=0, atol=6 * 6 * 2.0 ** -23)
                assert np.abs(both[2]).max() > 0
