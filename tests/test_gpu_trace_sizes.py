"""Closest-hit batches whose sizes do not fill a warp or a block: each ray's
result is the one it has in a larger batch, and nothing past the batch is
written."""
import numpy as np
import pytest

from conftest import random_rays
from cudart_gb300 import GB300Scene, _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 4097])
def test_partial_warps(cuda, n, fmt):
    g = GB300Scene(scenes.mixed_mid(subdiv=3), node_format=fmt)
    rays = cuda.from_numpy(random_rays(5000, 21)).cuda()
    idx, t, uv = (x.cpu().numpy() for x in g.trace_closest(rays))
    face = cuda.full((n + 64,), -7, dtype=cuda.int32, device="cuda")
    dist = cuda.full((n + 64,), -7.0, dtype=cuda.float32, device="cuda")
    stream = cuda.cuda.current_stream().cuda_stream
    assert _lib.load().crt_trace_closest(g.handle, rays.data_ptr(), n, face.data_ptr(), dist.data_ptr(), None, stream) == 0
    face, dist = face.cpu().numpy(), dist.cpu().numpy()
    assert np.array_equal(face[:n], idx[:n]) and np.array_equal(dist[:n], t[:n])
    assert (face[n:] == -7).all() and (dist[n:] == -7.0).all()
    nodes, tris = (x.cpu().numpy() for x in g.trace_counts(rays[:n]))
    assert len(nodes) == n and (nodes >= 1).all() and (tris[idx[:n] >= 0] >= 1).all()
