"""Material ids and emitters, which scene creation looks over on the device:
the emitters found are the ones listed, in face order, at face counts around a
warp's 32; of several faults the first in the order ids, emitters, textures,
coordinates is the one reported, with a device and without."""
import dataclasses

import numpy as np
import pytest

from cudart_gb300 import GB300Renderer, GB300Scene, scenes
from cudart_gb300._lib import CrtError


def _scene(n, emitters, seed=1):
    rng = np.random.default_rng(seed)
    base = scenes.cornell_box(width=16, height=16)
    pos = (rng.uniform(-0.9, 0.9, (n, 1, 3)) + rng.uniform(-0.3, 0.3, (n, 3, 3))).astype(np.float32)
    ids = np.zeros(n, np.uint32)
    ids[emitters] = 1
    return dataclasses.replace(base, positions=pos, normals=np.ones((n, 3, 3), np.float32),
                               uvs=np.zeros((n, 3, 2), np.float32), material_ids=ids,
                               materials=[base.materials[0], base.materials[3]], groups=[])


EMPTY = [np.zeros((0, 4, 4), np.uint8)]


@pytest.mark.parametrize("textures", [[], EMPTY])
@pytest.mark.parametrize("face", [0, 31, 32, 69])
def test_lowest_bad_id_is_reported_first(face, textures):
    sc = _scene(70, [])                       # no emitter either
    sc.material_ids[face:] = 2
    with pytest.raises(CrtError, match=f"material id out of range at face {face}"):
        GB300Scene(dataclasses.replace(sc, textures=textures))


@pytest.mark.parametrize("textures", [[], EMPTY])
def test_no_emitter_is_reported_before_textures(textures):
    with pytest.raises(CrtError, match="no emissive triangles"):
        GB300Scene(dataclasses.replace(_scene(70, []), textures=textures))


def test_empty_texture():
    with pytest.raises(CrtError, match="empty texture"):
        GB300Scene(dataclasses.replace(_scene(70, [3]), textures=EMPTY))


@pytest.mark.gpu
def test_bad_id_is_reported_before_coordinates(cuda):
    sc = _scene(70, [3])
    sc.positions[5, 0, 0] = np.nan
    sc.material_ids[50] = 9
    with pytest.raises(CrtError, match="material id out of range at face 50"):
        GB300Scene(sc, builder="gpu")


@pytest.mark.gpu
@pytest.mark.parametrize("builder", ["host", "gpu"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 1000])
def test_emitters_are_found_in_face_order(cuda, n, builder):
    rng = np.random.default_rng(n)
    for emitters in (np.arange(n), np.array([0]), np.array([n - 1]), np.unique(rng.integers(0, n, max(n // 3, 1)))):
        sc = _scene(n, emitters)
        found, listed = GB300Scene(sc, builder=builder), GB300Scene(sc, lights=emitters, builder=builder)
        assert found.info.num_lights == len(emitters)
        assert found.info.lights_area == listed.info.lights_area
        a, b = (GB300Renderer(g, 16, 16, 2, max_depth=3, seed=4) for g in (found, listed))
        a.render(), b.render()
        assert np.array_equal(a.accum(), b.accum())
