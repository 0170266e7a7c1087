"""Passes and tiles of few paths run each path in one thread, with 1 to 32
paths per warp: sums and ray counts equal the plain kernel's and the wave
form's at every size around the choices."""
import ctypes as C

import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, _lib, camera_from_json, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (7, 5, 3), (61, 67, 1), (64, 65, 2), (129, 127, 4), (362, 362, 1),
                                     (512, 256, 1),       # 2^17 paths: the last on the path kernel
                                     (363, 362, 1)])      # the first beyond
def test_small_pass_equals_plain_and_wave(cuda, w, h, spp, fmt):
    sc = scenes.feature_mix(width=w, height=h)
    g = GB300Scene(sc, node_format=fmt)
    plain = GB300Renderer(g, w, h, spp, max_depth=6, mode="megakernel")
    small = GB300Renderer(g, w, h, spp, max_depth=6, mode="wavefront")
    wave = GB300Renderer(g, w, h, spp, max_depth=6, mode="wavefront", wave_paths=1 << 16)
    for r in (plain, small, wave):
        r.render()
        r.render(1)                      # the next pass continues with the next sample
    assert np.array_equal(small.accum(), plain.accum())
    assert np.array_equal(small.accum(), wave.accum())
    assert small.ray_counts() == wave.ray_counts() == plain.ray_counts()
    small.restart(0)
    small.render(spp + 1)                # another size on the same handle
    assert np.array_equal(small.accum(), plain.accum())


@pytest.mark.parametrize("pixel0,count,nspp", [(0, 1, 1), (5, 31, 1), (17, 2090, 2), (3, 4096, 16), (100, 3797, 11)])
def test_tile_ranges(cuda, pixel0, count, nspp):
    """Only the tile's pixels change, and they equal the plain kernel's sums."""
    sc = scenes.mixed_mid(width=96, height=64, subdiv=2)
    g = GB300Scene(sc)
    cam = camera_from_json(sc.camera, sc.width, sc.height)
    acc = cuda.full((sc.width * sc.height, 4), 0.5, dtype=cuda.float32, device="cuda")
    opts = _lib.RenderOptions()
    _lib.load().crt_render_options_default(C.byref(opts))
    opts.max_depth = 8
    stream = cuda.cuda.current_stream().cuda_stream
    assert _lib.load().crt_render_tile_noalloc(g.handle, C.byref(cam), sc.width, sc.height, C.byref(opts), pixel0,
                                               count, 0, nspp, acc.data_ptr(), stream) == 0
    r = GB300Renderer(g, sc.width, sc.height, nspp, max_depth=8)
    r.load_accum(np.full((sc.width * sc.height, 3), 0.5, np.float32), 0)
    r.render()
    want, got = r.accum(), acc[:, :3].cpu().numpy()
    inside = np.arange(sc.width * sc.height)
    inside = (inside >= pixel0) & (inside < pixel0 + count)
    assert np.array_equal(got[inside], want[inside])
    assert (got[~inside] == 0.5).all() and (acc[:, 3] == 0.5).all()
