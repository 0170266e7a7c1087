"""A handle's first pass allocates and clears its wave sets while other
handles' kernels fill the GPU: its image must not depend on when that clearing
runs."""
import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, scenes

pytestmark = pytest.mark.gpu


def test_first_pass_beside_another_handles_work(cuda):
    sc = scenes.mixed_mid(width=256, height=144, subdiv=3)
    g = GB300Scene(sc)
    alone = GB300Renderer(g, 256, 144, 32, max_depth=6, mode="megakernel")
    alone.render()
    want = alone.accum()
    busy = GB300Renderer(g, 256, 144, 2048, max_depth=6, mode="wavefront", seed=9)
    for wave_paths in (1 << 16, 1 << 18, 0):
        busy.restart(0)
        busy.render()                     # milliseconds of persistent kernels
        first = GB300Renderer(g, 256, 144, 32, max_depth=6, mode="wavefront", wave_paths=wave_paths)
        first.render()                    # queued while they run
        assert np.array_equal(first.accum(), want)
    busy.synchronize()
