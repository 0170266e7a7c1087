"""GPU BVH builds at triangle counts around the clustering's block and halo
sizes (256 clusters, 3 and 6 on either side) and the smallest trees: the tree's
invariants, and closest hits equal to brute force."""
import dataclasses

import numpy as np
import pytest

import oracle
from conftest import random_rays
from cudart_gb300 import GB300Scene, scenes
from test_bvh_host import check_tree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 250, 253, 256, 257, 259, 262, 263, 511, 515, 1024, 4099, 70001])
def test_sizes(cuda, n, width):
    rng = np.random.default_rng(n)
    pos = (rng.uniform(-0.9, 0.9, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))).astype(np.float32)
    light = scenes.cornell_box()
    mats = [light.materials[0], dataclasses.replace(light.materials[3])]
    ids = np.zeros(n, np.uint32)
    ids[n // 2] = 1                                     # the one emitter, anywhere
    sc = dataclasses.replace(light, positions=pos, normals=np.ones((n, 3, 3), np.float32),
                             uvs=np.zeros((n, 3, 2), np.float32), material_ids=ids, materials=mats, groups=[])
    g = GB300Scene(sc, builder="gpu", bvh_width=width)
    nodes, tris = g.export_bvh()
    check_tree(pos, nodes, tris, g.info.max_depth, width)
    assert g.info.num_nodes == len(nodes) and g.info.num_lights == 1
    rays = random_rays(1500 if n < 5000 else 300, 5)
    idx, t, _ = g.trace_closest(cuda.from_numpy(rays).cuda())
    oi, ot, _ = oracle.OracleScene(sc).closest_hit(rays, brute=True)
    assert np.array_equal(idx.cpu().numpy(), oi) and np.array_equal(t.cpu().numpy(), ot)
