"""Passes of few paths take the path kernel unless a wave size or a flag asks for
the wave form; the options the tuner returns do not, where its trials kept the
default wave size.  Which form ran shows in the memory that it took: a wave set
of 2^16 paths is 140 bytes a path, the path kernel 16."""
import ctypes as C
import gc

import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, _lib, camera_from_json, scenes

pytestmark = pytest.mark.gpu
W, H = 64, 48
WAVE_SET = 140 << 16


def _taken(cuda, g, **kw):
    """Device memory that a handle takes for a pass of 12,288 paths, and its image."""
    gc.collect()
    r = GB300Renderer(g, W, H, 4, max_depth=5, **kw)
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    r.render()
    r.synchronize()
    return free - cuda.cuda.mem_get_info()[0], r.accum()


@pytest.fixture
def scene(cuda):
    g = GB300Scene(scenes.cornell_box(width=W, height=H))
    for kw in (dict(), dict(wave_paths=1 << 16)):       # kernels loaded before memory is looked at
        _taken(cuda, g, mode="wavefront", **kw)
    return g


@pytest.mark.parametrize("shape,sets", [(dict(), 0), (dict(block_size=128), 0), (dict(stack_depth=8, queue_chunk=32), 0),
                                        (dict(wave_sets=4), 0), (dict(block_size=64, wave_sets=2), 0),
                                        (dict(wave_paths=1 << 16), 4), (dict(wave_paths=1 << 16, wave_sets=2), 2),
                                        (dict(flags=16), 4)])
def test_what_asks_for_the_wave_form(cuda, scene, shape, sets):
    taken, image = _taken(cuda, scene, mode="wavefront", **shape)
    plain = GB300Renderer(scene, W, H, 4, max_depth=5)
    plain.render()
    assert np.array_equal(image, plain.accum())
    if sets:
        assert taken >= sets * WAVE_SET
    else:
        assert taken < WAVE_SET


def test_tuned_options(cuda, scene):
    """Room for the default wave size alone: the trials cannot choose another."""
    L = _lib.load()
    start, p, res = _lib.RenderOptions(), _lib.TuneParams(), _lib.TuneResult()
    L.crt_render_options_default(C.byref(start))
    start.max_depth = 5
    L.crt_tune_params_default(C.byref(p))
    p.repeats, p.rounds, p.tune_bvh_width, p.max_wave_bytes = 1, 1, 0, 5 * WAVE_SET
    cam = camera_from_json(scene.arrays.camera, W, H)
    assert L.crt_autotune(scene.handle, C.byref(cam), W, H, C.byref(start), C.byref(p), C.byref(res)) == 0
    assert res.options.wave_paths == 0 and res.options.wave_sets > 0 and res.options.block_size > 0
    res.options.flags = 0
    taken, _ = _taken(cuda, scene, options=res.options)
    assert taken < WAVE_SET
    start.wave_paths = 1 << 16                          # the caller's own choice stays
    assert L.crt_autotune(scene.handle, C.byref(cam), W, H, C.byref(start), C.byref(p), C.byref(res)) == 0
    assert res.options.wave_paths == 1 << 16
