"""The clearance that planes give a triangle pair of the clearance cache, under rotations of the bodies as well as
shifts, far from the origin, and on slivers: no segment while the motion, measured as the cache measures it, stays
below the clearance."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_plane_margin_cpu import sliver_pairs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _pairs(rng, n, scale):
    T = rng.normal(size=(n, 2, 3, 3)) * scale
    k = np.arange(n) % 6
    T[k == 0, 1] += rng.normal(size=(np.sum(k == 0), 1, 3)) * scale * 2
    T[k == 1, 1] = T[k == 1, 0] + rng.normal(size=(np.sum(k == 1), 1, 3)) * scale * 1e-2       # close and parallel
    T[k == 2, 1, :, 2] = T[k == 2, 0].max(axis=(1, 2))[:, None] + 10.0 ** rng.uniform(-6, -1, size=(np.sum(k == 2), 1)) * scale
    T[k == 3, :, :, 2] *= 1e-5                                                                  # nearly one plane
    T[k == 4, 0, 2] = 0.5 * (T[k == 4, 0, 0] + T[k == 4, 0, 1]) + rng.normal(size=(np.sum(k == 4), 3)) * scale * 1e-5
    T[k == 5] = sliver_pairs(rng, np.sum(k == 5), scale)
    return T


@pytest.mark.parametrize("scale", [1e-4, 1e-3, 1.0, 100.0])
@pytest.mark.parametrize("far", [0.0, 1.0, 1e3])
def test_no_segment_within_the_clearance(tmp_path, scale, far):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path / "plane_motion_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "zedm-x_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "plane_motion_check.cpp")], check=True, timeout=300)
    rng = np.random.default_rng([int(scale * 1e4), int(far)])
    n = 40000
    T = _pairs(rng, n, scale)
    # the bodies' frames: each triangle's origin some way off, so that a turn moves it, and turned
    x = T.mean(axis=2) + rng.normal(size=(n, 2, 3)) * scale * 10.0 ** rng.uniform(-2, 1, size=(n, 2, 1))
    q = rng.normal(size=(n, 2, 4))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    local = T - x[:, :, None]
    u, w = -q[:, :, None, 1:], q[:, :, None, :1]
    h = 2.0 * np.cross(u, local)
    local = local + w * h + np.cross(u, h)
    x = x + rng.uniform(-1, 1, size=(n, 1, 3)) * far
    motion = rng.uniform(-1, 1, size=(n, 2, 4))
    motion[::3, :, 3] = 0.0
    motion[1::3, :, 3] = 1.0
    rows = np.concatenate([local.reshape(n, 18), np.concatenate([x, q], 2).reshape(n, 14), motion.reshape(n, 8)], 1)
    text = "\n".join(" ".join("%016x" % v for v in row) for row in np.ascontiguousarray(rows).view(np.uint64))
    p = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=300)
    got, held, wrong = (int(v) for v in p.stdout.split())
    assert got == n and held > 1000
    assert wrong == 0
