"""The clearance a triangle pair gets from the triangles' planes: after rigid moves of both that add up to less than
it, tri_tri finds no segment -- on pairs far apart, close, coplanar, slivers, and about the tolerance off a plane."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("scale", [1e-4, 1e-3, 1.0, 100.0])
def test_no_segment_within_the_clearance(tmp_path, scale):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path / "plane_clear_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "zedm-x_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "plane_clear_check.cpp")], check=True, timeout=300)
    rng = np.random.default_rng(int(scale * 1e4) + 1)
    n = 40000
    T = rng.normal(size=(n, 2, 3, 3)) * scale
    k = np.arange(n) % 5
    T[k == 0, 1] += rng.normal(size=(np.sum(k == 0), 1, 3)) * scale * 2
    T[k == 1, 1] = T[k == 1, 0] + rng.normal(size=(np.sum(k == 1), 1, 3)) * scale * 1e-2      # close and parallel
    T[k == 2, 1, :, 2] = T[k == 2, 0].max(axis=(1, 2))[:, None] + 10.0 ** rng.uniform(-8, -1, size=(np.sum(k == 2), 1)) * scale
    T[k == 3, :, :, 2] *= 1e-6                                                                 # nearly one plane
    T[k == 4, 0, 2] = 0.5 * (T[k == 4, 0, 0] + T[k == 4, 0, 1]) + rng.normal(size=(np.sum(k == 4), 3)) * scale * 1e-5
    rows = np.concatenate([T.reshape(n, 18), rng.uniform(-1, 1, size=(n, 6))], 1)
    text = "\n".join(" ".join("%016x" % x for x in row) for row in np.ascontiguousarray(rows).view(np.uint64))
    p = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=300)
    got, held, wrong = (int(x) for x in p.stdout.split())
    assert got == n and held > 4000
    assert wrong == 0
