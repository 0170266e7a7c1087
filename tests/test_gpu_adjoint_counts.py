"""Ray counts of an adjoint pass: the rays of both of its traces, whether the
second traces them again (17 bounces) or reads the first's hits (up to 16)."""
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, 4, 16])          # window sort, octant queues, neither
@pytest.mark.parametrize("depth", [1, 6, 16, 17])
def test_both_traces_count(cuda, depth, flags):
    sc = scenes.material_inversion(width=61, height=47)
    g = GB300Scene(sc)
    n = len(sc.materials)
    kw = dict(max_depth=depth, seed=5, mode="wavefront", wave_paths=1 << 13, flags=flags)   # several waves a set
    frame = GB300Renderer(g, 61, 47, 24, **kw)
    frame.render()
    ext, shadow = frame.ray_counts()
    assert ext > 61 * 47 * 24 and shadow > 0 or depth == 1
    weights = cuda.rand((61 * 47, 4), device="cuda")
    kd, ka = cuda.zeros((n, 3), device="cuda"), cuda.zeros((n, 3), device="cuda")
    cuda.cuda.synchronize()
    r = GB300Renderer(g, 61, 47, 24, **kw)
    r.adjoint(0, 24, weights.data_ptr(), kd.data_ptr(), ka.data_ptr())
    assert r.ray_counts() == (2 * ext, 2 * shadow)
