"""The adjoint with little device memory left: the record of the primal trace is
optional and must not take the room of the buffers the adjoint needs.

Two wave sets of 2^20 paths at depth 16: 48 MiB each of needed buffers (32 more
for the exact roulette's history) and 260 MiB each of record.  The rest of the
device's memory is held by one tensor meanwhile."""
import gc

import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, scenes

pytestmark = pytest.mark.gpu
MIB = 1 << 20
NEEDED, HISTORY, RECORD = 48 * MIB, 32 * MIB, 260 * MIB     # per set


def _handle():
    sc = scenes.material_inversion(width=61, height=47)
    g = GB300Scene(sc)
    r = GB300Renderer(g, 61, 47, 8, max_depth=16, seed=5, mode="wavefront", wave_paths=1 << 20, wave_sets=2)
    r.render(1)
    r.synchronize()
    return len(sc.materials), r


def _grads(cuda, r, n, weights, exact=False):
    kd, ka = cuda.zeros((n, 3), device="cuda"), cuda.zeros((n, 3), device="cuda")
    cuda.cuda.synchronize()
    r.adjoint(0, 8, weights.data_ptr(), kd.data_ptr(), ka.data_ptr(), exact_roulette=exact)
    r.synchronize()
    return cuda.cat([kd, ka]).double().cpu().numpy()


def _free(cuda):
    cuda.cuda.synchronize()
    return cuda.cuda.mem_get_info()[0]


def _hold_all_but(cuda, room):
    hold = cuda.empty(_free(cuda) - room, dtype=cuda.uint8, device="cuda")
    assert room - 32 * MIB <= _free(cuda) <= room
    return hold


@pytest.fixture
def weights(cuda):
    gc.collect()                                   # earlier tests' handles, not in the middle of this one
    yield cuda.rand((61 * 47, 4), generator=cuda.Generator("cuda").manual_seed(1), device="cuda")
    cuda.cuda.empty_cache()


def _same(got, want):
    """Sums of the same FP32 terms, rounded once per block and once per call (2^-24 each)."""
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


def test_record_leaves_room_for_what_every_set_needs(cuda, weights):
    n, plenty = _handle()
    before = _free(cuda)
    want = _grads(cuda, plenty, n, weights)
    assert before - _free(cuda) >= 2 * (NEEDED + RECORD)          # with room, it is kept
    del plenty
    n, r = _handle()
    # one set's buffers and record would fit, and the other set's buffers no more
    hold = _hold_all_but(cuda, NEEDED + RECORD + NEEDED // 2)
    got = [_grads(cuda, r, n, weights) for _ in range(2)]
    assert _free(cuda) >= 100 * MIB                               # no record
    del hold
    for g in got:
        _same(g, want)


def test_record_leaves_as_much_again(cuda, weights):
    n, r = _handle()
    hold = _hold_all_but(cuda, 2 * NEEDED + 3 * RECORD)           # fits, and would leave half of its size
    want = _grads(cuda, r, n, weights)
    assert _free(cuda) >= 2 * RECORD
    del hold
    cuda.cuda.empty_cache()
    n, plenty = _handle()
    _same(_grads(cuda, plenty, n, weights), want)


def test_record_gives_way_to_the_exact_roulette_history(cuda, weights):
    n, r = _handle()
    before = _free(cuda)
    want = _grads(cuda, r, n, weights)
    assert before - _free(cuda) >= 2 * (NEEDED + RECORD)
    hold = _hold_all_but(cuda, HISTORY)                           # less than the two sets' histories
    exact = _grads(cuda, r, n, weights, exact=True)
    _same(_grads(cuda, r, n, weights), want)
    del hold
    cuda.cuda.empty_cache()
    n, plenty = _handle()
    _same(exact, _grads(cuda, plenty, n, weights, exact=True))
