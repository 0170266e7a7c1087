"""Few paths, walked in 8x4 tiles where whole 4-row bands of a width divisible
by 8 lie in the range and in rows otherwise, with as many paths per warp as
leave one resident wave (1 to 32, any number): sums equal the plain kernel's."""
import ctypes as C

import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, _lib, camera_from_json, scenes

pytestmark = pytest.mark.gpu


# ranges that start on a row (tiled part, then rows), inside one, and shorter than a band
@pytest.mark.parametrize("pixel0,count,nspp", [(0, 384, 3), (192, 384 * 3 + 17, 2), (96, 383, 5), (96, 768, 80),
                                               (97, 768, 4), (0, 6144, 10)])
@pytest.mark.parametrize("width", [96, 92])
def test_ranges(cuda, width, pixel0, count, nspp):
    sc = scenes.mixed_mid(width=width, height=64, subdiv=2)
    npix = sc.width * sc.height
    count = min(count, npix - pixel0)
    g = GB300Scene(sc)
    cam = camera_from_json(sc.camera, sc.width, sc.height)
    acc = cuda.zeros((npix, 4), dtype=cuda.float32, device="cuda")
    opts = _lib.RenderOptions()
    _lib.load().crt_render_options_default(C.byref(opts))
    opts.max_depth = 8
    assert _lib.load().crt_render_tile_noalloc(g.handle, C.byref(cam), sc.width, sc.height, C.byref(opts), pixel0,
                                               count, 0, nspp, acc.data_ptr(),
                                               cuda.cuda.current_stream().cuda_stream) == 0
    r = GB300Renderer(g, sc.width, sc.height, nspp, max_depth=8)
    r.render()
    want, got = r.accum(), acc[:, :3].cpu().numpy()
    assert np.array_equal(got[pixel0:pixel0 + count], want[pixel0:pixel0 + count])
    assert (got[:pixel0] == 0).all() and (got[pixel0 + count:] == 0).all()


@pytest.mark.parametrize("w,h,spp", [(8, 4, 1), (16, 7, 3), (96, 33, 1), (96, 65, 8), (256, 250, 2)])
def test_whole_views(cuda, w, h, spp):
    g = GB300Scene(scenes.feature_mix(width=w, height=h), node_format="f32")
    plain = GB300Renderer(g, w, h, spp, max_depth=6, mode="megakernel")
    small = GB300Renderer(g, w, h, spp, max_depth=6, mode="wavefront")
    plain.render(), small.render()
    assert np.array_equal(small.accum(), plain.accum())
    assert small.ray_counts() == plain.ray_counts()
