"""The traversal kernels' change from batches to lane refill inside a launch:
queues just around the sizes where a warp decides, runs dry or refills its last
lanes give the plain kernel's sums and ray counts."""
import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, _lib, scenes

pytestmark = pytest.mark.gpu


def _scene(w, h):
    # one large ball of many triangles and bare walls: rays differ widely in
    # visits, so the warps do change over
    return scenes.mixed_mid(width=w, height=h, subdiv=4, seed=3)


@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("w,h,spp,wave_paths", [(640, 360, 4, 0),         # several batches per warp
                                                (97, 61, 53, 1 << 18),    # an odd queue length
                                                (64, 32, 1, 2048),        # fewer entries than lanes on the chip
                                                (33, 1, 1, 33)])          # one warp and one lane
@pytest.mark.parametrize("chunk", [0, 128])
def test_sums_and_counts(cuda, w, h, spp, wave_paths, chunk, fmt):
    g = GB300Scene(_scene(w, h), node_format=fmt)
    plain = GB300Renderer(g, w, h, spp, max_depth=8)
    want = None
    for kw in (dict(), dict(flags=_lib.FLAG_LANE_REFILL), dict(flags=_lib.FLAG_LANE_REFILL, refill_busy=1),
               dict(flags=_lib.FLAG_SPLIT_LEAF)):
        r = GB300Renderer(g, w, h, spp, max_depth=8, mode="wavefront", wave_paths=wave_paths or 1 << 20,
                          queue_chunk=chunk, **kw)
        r.render()
        if want is None:
            plain.render()
            want = plain.accum()
        assert np.array_equal(r.accum(), want), kw
        assert r.ray_counts() == plain.ray_counts(), kw
