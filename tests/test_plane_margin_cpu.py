"""The triangle stage's plane test on triangles whose computed plane leans: slivers of 1e-16 to 1e-5 of their length
cut by nearly coplanar triangles, at sizes from 1e-3 to 1e5, in the mesh frame's own place, rotated there, and placed
far away.  No pair that has a segment is ruled out, and ordinary pairs that lie apart still are."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# one segment, 1.0e-5 long: A lies 4.3e-8 beyond B's computed plane, from which B's own third corner stands 1.5e-7
LOST = np.array([[(0.15385935367133904, 0.1088033284441523, 0.12244409448146336),
                  (0.10222259118064242, 0.10231782126444401, 0.14202125563078161),
                  (0.16978377528197966, 0.085883818951380003, 0.066060708668352494)],
                 [(0.33554890505040869, 0.24346607373505155, 0.27951959369516527),
                  (-0.33554890505040869, -0.24346607373505155, -0.27951959369516527),
                  (-0.2896471982147098, -0.21016091879317533, -0.24128246606741849)]])


def sliver_pairs(rng, n, size):
    """(n, 2, 3, 3): a sliver of up to `size` along u, `th` wide along v, and a triangle about a point of it whose
    extent along the sliver's normal w is 1e-9 to 1 of the rest, lifted off along w by as little."""
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = np.cross(u, rng.normal(size=(n, 3)))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    w = np.cross(u, v)
    L = size * 10.0 ** rng.uniform(-1, 0, size=(n, 1))
    th = L * 10.0 ** rng.uniform(-16, -5, size=(n, 1))
    B = np.stack([u * L, -u * L, u * L * rng.uniform(-0.96, 0.96, size=(n, 1)) + v * th], 1)
    c = u * L * rng.uniform(-0.9, 0.9, size=(n, 1)) + v * th * rng.uniform(-1, 2, size=(n, 1))
    r = L * 10.0 ** rng.uniform(-4, 0, size=(n, 1))
    g = rng.normal(size=(n, 3, 3))
    g[:, :, 2] *= 10.0 ** rng.uniform(-9, 0, size=(n, 1))
    A = c[:, None] + r[:, None] * (g[:, :, :1] * u[:, None] + g[:, :, 1:2] * v[:, None] + g[:, :, 2:] * w[:, None])
    A += (w * 10.0 ** rng.uniform(-16, -3, size=(n, 1)) * L * rng.choice([-1, 0, 1], size=(n, 1)))[:, None]
    T = np.stack([A, B], 1)
    swap = rng.random(n) < 0.5
    T[swap] = T[swap][:, ::-1]
    return T


def _run(tmp_path, T, pose):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path / "plane_margin_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "zedm-x_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "plane_margin_check.cpp")], check=True, timeout=300)
    rows = np.ascontiguousarray(np.concatenate([T.reshape(len(T), 18), pose], 1))
    text = "\n".join(" ".join("%016x" % x for x in row) for row in rows.view(np.uint64))
    p = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=300)
    return [int(x) for x in p.stdout.split()]


@pytest.mark.parametrize("size", [1e-3, 0.1, 1.0, 10.0, 1e3, 1e5])
@pytest.mark.parametrize("place", ["own", "rotated", "far"])
def test_no_segment_of_a_sliver_is_ruled_out(tmp_path, size, place):
    n = 40000
    rng = np.random.default_rng([int(size * 1e3), ["own", "rotated", "far"].index(place)])
    pose = np.zeros((n, 7))
    pose[:, 3] = 1.0
    if place != "own":
        pose[:, 3:] = rng.normal(size=(n, 4))
    if place == "far":
        pose[:, :3] = rng.uniform(-1, 1, size=(n, 3)) * 10.0 ** rng.uniform(-2, 4, size=(n, 1))
    got, seg, _, wrong = _run(tmp_path, sliver_pairs(rng, n, size), pose)
    assert got == n and seg > 1000
    assert wrong == 0


def test_the_pair_that_was_lost(tmp_path):
    pose = np.zeros((2, 7))
    pose[:, 3] = 1.0
    assert _run(tmp_path, np.stack([LOST, LOST[::-1]]), pose) == [2, 2, 0, 0]


@pytest.mark.parametrize("scale", [1e-3, 1.0, 100.0])
def test_ordinary_pairs_are_still_ruled_out(tmp_path, scale):
    """Triangles on both sides of a gap of 1e-4 of their size: the margin is far below it."""
    n = 20000
    rng = np.random.default_rng(int(scale * 1e3))
    T = rng.normal(size=(n, 2, 3, 3))
    T[:, 0, :, 2] = 0.0
    T[:, 1, :, 2] = np.abs(T[:, 1, :, 2]) + 1e-4
    pose = np.concatenate([rng.uniform(-1, 1, size=(n, 3)) * scale, rng.normal(size=(n, 4))], 1)
    got, seg, out, wrong = _run(tmp_path, T * scale, pose)
    assert got == n and seg == 0 and wrong == 0
    assert out > 0.99 * n
