"""The device node encodings: rounding of the quantised planes (host code, no
GPU), and closest hits against brute force on geometry that stresses them."""
import dataclasses
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import FLT_MAX, ROOT
from cudart_gb300 import scenes


def test_plane_rounding_and_slots(tmp_path):
    exe = str(tmp_path / "node_encoding")
    src = os.path.join(ROOT, "tests", "c", "node_encoding.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O2", "-ffp-contract=off", src, "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout.startswith("ok "), p.stdout


def _scene(kind):
    """A light plus test triangles: far from the origin, tiny, or with an axis of no extent."""
    sc = scenes.mixed_mid(subdiv=2)
    p = sc.positions.astype(np.float64)
    if kind == "far":
        p = p + np.array([4096.0, -512.0, 1024.0])
    elif kind == "tiny":
        p = p * 2.0 ** -6
    elif kind == "flat":
        p = p.copy()
        p[12:, :, 2] = 0.25
    elif kind == "stretched":
        p = p * np.array([1000.0, 1.0, 0.01])
    return dataclasses.replace(sc, positions=p.astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("builder", ["host", "gpu"])
@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("kind", ["far", "tiny", "flat", "stretched"])
def test_closest_hits_on_awkward_boxes(cuda, kind, fmt, builder):
    """Origins on and around the bounds; directions random, axis-parallel and
    nearly axis-parallel.  Index and distance equal the brute force's, exactly."""
    import oracle
    from cudart_gb300 import GB300Scene
    sc = _scene(kind)
    rng = np.random.default_rng(11)
    n = 6000
    pts = sc.positions.reshape(-1, 3)
    lo, hi = pts.min(0), pts.max(0)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = lo + (hi - lo) * rng.uniform(-0.1, 1.1, (n, 3))
    rays[: n // 3, :3] = pts[rng.integers(0, len(pts), n // 3)]
    target = sc.positions[rng.integers(0, sc.n_tris, n)].mean(1)
    d = target - rays[:, :3] + rng.normal(size=(n, 3)) * (hi - lo) * 0.05
    d[: n // 4] = np.eye(3)[rng.integers(0, 3, n // 4)] * rng.choice([-1.0, 1.0], (n // 4, 1))
    d[n // 4: n // 3] += 1e-6 * rng.normal(size=(n // 3 - n // 4, 3))
    rays[:, 4:7] = d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)
    rays[:, 3], rays[:, 7] = 1e-5, FLT_MAX
    g = GB300Scene(sc, node_format=fmt, builder=builder)
    idx, t, _ = g.trace_closest(cuda.from_numpy(rays).cuda())
    oi, ot, _ = oracle.OracleScene(sc).closest_hit(rays, brute=True)
    assert (oi >= 0).mean() > 0.2
    assert np.array_equal(idx.cpu().numpy(), oi)
    assert np.array_equal(t.cpu().numpy(), ot)
