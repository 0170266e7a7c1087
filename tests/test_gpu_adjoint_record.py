"""The adjoint replay with and without the primal trace's record of hits and
visibilities (up to 16 bounces it is kept; beyond, the replay traces again)."""
import numpy as np
import pytest

import oracle
from cudart_gb300 import GB300Renderer, GB300Scene, scenes

pytestmark = pytest.mark.gpu


def _grads(torch, r, n_mats, a4, spp0, spp):
    gkd = torch.zeros((n_mats, 3), dtype=torch.float32, device="cuda")
    gka = torch.zeros((n_mats, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    r.adjoint(spp0, spp, a4.data_ptr(), gkd.data_ptr(), gka.data_ptr())
    r.synchronize()
    return gkd.cpu().numpy().astype(np.float64), gka.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("depth", [1, 2, 16, 17])
def test_matches_fp64_reference_on_either_side_of_the_record(cuda, depth):
    """As the adjoint's own reference test: relative error of the significant
    gradients (FP32 path arithmetic against FP64)."""
    sc = scenes.material_inversion(width=48, height=48)
    adj = np.random.default_rng(2).uniform(0.5, 1.5, (48 * 48, 3)).astype(np.float32)
    a4 = cuda.zeros((48 * 48, 4), dtype=cuda.float32, device="cuda")
    a4[:, :3] = cuda.from_numpy(adj).cuda()
    r = GB300Renderer(GB300Scene(sc), 48, 48, 16, max_depth=depth, seed=5, mode="wavefront")
    got = _grads(cuda, r, len(sc.materials), a4, 0, 16)
    ref = oracle.OracleScene(sc).adjoint(oracle.make_camera(sc.camera, 48, 48), 5, 16, depth, adj)
    for g, e in zip(got, ref):
        sig = np.abs(e) > 1e-3 * np.abs(e).max()
        rel = np.abs(g - e)[sig] / np.abs(e)[sig]
        assert np.median(rel) < 1e-4 and rel.max() < 1e-2


def test_several_waves_and_calls_add_up(cuda):
    """Small waves (several per set) and two calls into the same buffers equal
    one call over all samples: sums of the same FP32 terms, rounded once per block
    and once per call (2^-24 each, far below 1e-5)."""
    sc = scenes.material_inversion(width=61, height=47)
    a4 = cuda.rand((61 * 47, 4), device="cuda")
    g = GB300Scene(sc)
    n = len(sc.materials)
    whole = GB300Renderer(g, 61, 47, 24, max_depth=5, seed=5, mode="wavefront")
    parts = GB300Renderer(g, 61, 47, 24, max_depth=5, seed=5, mode="wavefront", wave_paths=1 << 12)
    want = _grads(cuda, whole, n, a4, 0, 24)
    gkd = cuda.zeros((n, 3), device="cuda")
    gka = cuda.zeros((n, 3), device="cuda")
    cuda.cuda.synchronize()
    parts.adjoint(0, 7, a4.data_ptr(), gkd.data_ptr(), gka.data_ptr())
    parts.adjoint(7, 17, a4.data_ptr(), gkd.data_ptr(), gka.data_ptr())
    parts.synchronize()
    for got, ref in ((gkd, want[0]), (gka, want[1])):
        got = got.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
