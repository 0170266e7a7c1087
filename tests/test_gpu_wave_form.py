"""The wave form on images of few paths.  A pass of few paths takes the path
kernel unless its wave size is asked for; these handles ask for one, so that
captured wave graphs, the window sort and narrow trees meet the wave kernels."""
import numpy as np
import pytest

from cudart_gb300 import CrtError, GB300Renderer, GB300Scene, scenes

pytestmark = pytest.mark.gpu
CRT_ERR_WATCHDOG = 5
WAVE = dict(mode="wavefront", wave_paths=1 << 14)      # several waves on every set


def _large():
    return scenes.large_textured(width=96, height=54, grid=64, tex_size=64, n_spheres=12, sphere_subdiv=2)


@pytest.mark.parametrize("wave_paths", [1 << 14, 1 << 18])
@pytest.mark.parametrize("builder", ["host", "gpu"])
def test_graphs_follow_a_rebuilt_tree(cuda, builder, wave_paths):
    sc = scenes.mixed_mid(width=128, height=72, subdiv=3)
    g = GB300Scene(sc, builder=builder)
    r = GB300Renderer(g, 128, 72, 4, max_depth=8, mode="wavefront", wave_paths=wave_paths)
    r.render()                                  # captures its wave graphs on the 8-wide tree
    r.render()                                  # replays them
    n8 = g.info.num_nodes
    g.set_bvh_width(4)
    assert g.info.bvh_width == 4 and g.info.num_nodes > n8
    r.render()                                  # must capture against the new nodes
    plain = GB300Renderer(GB300Scene(sc), 128, 72, 12, max_depth=8)
    plain.render()
    assert np.array_equal(r.accum(), plain.accum())


def test_adjoint_graphs_follow_a_rebuilt_tree(cuda):
    sc = scenes.material_inversion(width=64, height=48)
    weights = 0.5 + cuda.rand((64 * 48, 4), device="cuda")
    g, n = GB300Scene(sc), len(sc.materials)
    r = GB300Renderer(g, 64, 48, 8, max_depth=5, **WAVE)
    out = []
    for width in (8, 4):
        g.set_bvh_width(width)
        kd, ka = cuda.zeros((n, 3), device="cuda"), cuda.zeros((n, 3), device="cuda")
        cuda.cuda.synchronize()
        r.adjoint(0, 8, weights.data_ptr(), kd.data_ptr(), ka.data_ptr())
        r.synchronize()
        out.append(cuda.cat([kd, ka]).double().cpu().numpy())
    # the same FP32 terms; block sums in another order, rounded at 2^-24 each
    assert np.linalg.norm(out[1] - out[0]) <= 1e-5 * np.linalg.norm(out[0]) > 0


def test_graphs_follow_the_visit_limit(cuda):
    sc = scenes.feature_mix(width=48, height=32)
    g = GB300Scene(sc)
    want = GB300Renderer(g, sc.width, sc.height, 4, max_depth=6)
    want.render()
    r = GB300Renderer(g, sc.width, sc.height, 4, max_depth=6, **WAVE)
    r.render()                      # graphs captured under the default limit
    r.synchronize()
    g.set_visit_limit(2)            # root + one child: most rays run out
    r.reset()
    r.render()
    with pytest.raises(CrtError) as e:
        r.synchronize()
    assert e.value.status == CRT_ERR_WATCHDOG
    g.set_visit_limit(0)
    g.clear_errors()
    r.reset()
    r.render()
    assert np.array_equal(r.accum(), want.accum())


@pytest.mark.parametrize("flags", [0, 16, 4, 8])       # window sort (the default), warp order, octants, serial shadow
@pytest.mark.parametrize("fmt", ["q8", "f32"])
def test_window_sort(cuda, fmt, flags):
    """Four lights, a texture, mirrors and glass; many windows and partial last windows."""
    sc = _large()
    g = GB300Scene(sc, node_format=fmt)
    plain = GB300Renderer(g, sc.width, sc.height, 8, max_depth=8)
    plain.render()
    for wave_paths in (1 << 14, 1 << 16, 5000):
        r = GB300Renderer(g, sc.width, sc.height, 8, max_depth=8, mode="wavefront", wave_paths=wave_paths, flags=flags)
        r.render()
        assert np.array_equal(r.accum(), plain.accum()) and r.ray_counts() == plain.ray_counts()


@pytest.mark.parametrize("builder", ["host", "gpu"])
def test_four_wide_tree(cuda, builder):
    sc = scenes.mixed_mid(width=128, height=72, subdiv=3)
    plain = GB300Renderer(GB300Scene(sc), 128, 72, 8, max_depth=8)
    plain.render()
    r = GB300Renderer(GB300Scene(sc, builder=builder, bvh_width=4), 128, 72, 8, max_depth=8, **WAVE)
    r.render()
    assert np.array_equal(r.accum(), plain.accum())


def test_node_formats(cuda):
    sc = _large()
    out = []
    for fmt in ("q8", "f32"):
        r = GB300Renderer(GB300Scene(sc, node_format=fmt), sc.width, sc.height, 8, max_depth=8, **WAVE)
        r.render()
        out.append(r.accum())
    assert np.array_equal(out[0], out[1])


def test_reference_layout(cuda):
    sc = scenes.feature_mix(width=64, height=48)
    out = []
    for layout in (False, True):
        r = GB300Renderer(GB300Scene(sc, reference_layout=layout), sc.width, sc.height, 8, max_depth=6, **WAVE)
        r.render()
        out.append(r.accum())
    assert np.array_equal(out[0], out[1])


def test_resume_and_async_read(cuda):
    sc = scenes.cornell_box(width=64, height=48)
    g = GB300Scene(sc)
    full = GB300Renderer(g, 64, 48, 10, max_depth=5, **WAVE)
    full.render(10)
    part = GB300Renderer(g, 64, 48, 10, max_depth=5, **WAVE)
    part.render(4)
    early = cuda.empty(64 * 48 * 4, dtype=cuda.uint8).pin_memory()
    part.resolve_async(early)
    image = part.copy_image_bytes()              # the same staging memory, queued behind the copy
    resumed = GB300Renderer(g, 64, 48, 10, max_depth=5, **WAVE)
    resumed.load_accum(part.accum(), part.get_samples_rendered(), 0)
    resumed.render(6)
    part.render(6)
    assert np.array_equal(early.numpy().reshape(48, 64, 4), image)
    assert np.array_equal(resumed.accum(), full.accum()) and np.array_equal(part.accum(), full.accum())


def test_pixel_order_with_whole_images_per_wave(cuda):
    sc = scenes.cornell_box(width=64, height=48)
    g = GB300Scene(sc)
    plain = GB300Renderer(g, 64, 48, 6, max_depth=5)
    plain.render()
    for wave_paths in (64 * 48, 64 * 48 * 6, 1 << 16):
        r = GB300Renderer(g, 64, 48, 6, max_depth=5, mode="wavefront", wave_paths=wave_paths)
        r.render()
        assert np.array_equal(r.accum(), plain.accum())
