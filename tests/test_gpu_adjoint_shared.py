"""Gradients are added to the caller's arrays: several handles may add to the
same ones at once, and the two outputs may be one array.

The weights are positive, so every term of every sum is positive or zero and a
sum in another order differs by at most (terms) x 2^-24 of itself: 48 x 48 x 16
paths of at most 5 vertices, under 2^18 terms over all blocks, which add at most
2^13 each in FP32 before the FP64 totals: 2^-11.  A lost addend is a third of
the sum or more."""
import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, scenes

pytestmark = pytest.mark.gpu
SIDE, SPP = 48, 16


def _setup(cuda, handles):
    sc = scenes.material_inversion(width=SIDE, height=SIDE)
    g = GB300Scene(sc)
    weights = 0.5 + cuda.rand((SIDE * SIDE, 4), generator=cuda.Generator("cuda").manual_seed(3), device="cuda")
    rs = [GB300Renderer(g, SIDE, SIDE, SPP, max_depth=5, seed=7 + k, mode="wavefront", wave_paths=1 << 16)
          for k in range(handles)]
    return len(sc.materials), weights, rs


def _alone(cuda, r, n, weights):
    kd, ka = cuda.zeros((n, 3), device="cuda"), cuda.zeros((n, 3), device="cuda")
    cuda.cuda.synchronize()
    r.adjoint(0, SPP, weights.data_ptr(), kd.data_ptr(), ka.data_ptr())
    r.synchronize()
    return kd.double().cpu().numpy(), ka.double().cpu().numpy()


def test_handles_on_their_own_streams_add_to_one_pair_of_arrays(cuda):
    n, weights, rs = _setup(cuda, 3)
    single = [_alone(cuda, r, n, weights) for r in rs]
    want = [sum(s[k] for s in single) for k in range(2)]
    rounds = 20                                   # calls of the three handles end close together
    kd, ka = cuda.zeros((n, 3), device="cuda"), cuda.zeros((n, 3), device="cuda")
    cuda.cuda.synchronize()
    for _ in range(rounds):
        for r in rs:
            r.adjoint(0, SPP, weights.data_ptr(), kd.data_ptr(), ka.data_ptr())
    for r in rs:
        r.synchronize()
    for got, w in ((kd, want[0]), (ka, want[1])):
        assert (w >= 0).all() and w.max() > 0
        # 60 further FP32 additions into each element: 60 x 2^-24
        assert np.abs(got.double().cpu().numpy() / rounds - w).max() <= (2.0 ** -10) * w.max()


def test_one_array_for_both_outputs(cuda):
    n, weights, (r,) = _setup(cuda, 1)
    kd, ka = _alone(cuda, r, n, weights)
    both = cuda.zeros((n, 3), device="cuda")
    cuda.cuda.synchronize()
    r.adjoint(0, SPP, weights.data_ptr(), both.data_ptr(), both.data_ptr())
    r.synchronize()
    got = both.double().cpu().numpy()
    assert (kd > 0).any() and (ka > 0).any() and ((kd > 0) & (ka > 0)).any()
    assert np.allclose(got, kd + ka, rtol=2.0 ** -10, atol=0)
