"""The parts the triangle stage takes tri_tri apart into: candidates and join against the whole, to the bit, in both
arithmetics, and the plane test never rules out a pair that has a segment -- on triangle pairs that cross, touch,
share edges or corners, lie in one plane, are slivers, or miss each other by about point_in_tri's tolerance."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _pairs(rng, n, scale):
    T = rng.normal(size=(n, 2, 3, 3)) * scale
    T[:, 1] += rng.normal(size=(n, 1, 3)) * scale * 0.5
    k = np.arange(n) % 8
    T[k == 1, 1, 0] = T[k == 1, 0, 0]                                             # a shared corner
    T[k == 2, 1, :2] = T[k == 2, 0, :2]                                           # a shared edge
    T[k == 3, :, :, 2] = 0.0                                                      # one plane
    T[k == 4, 0, 2] = 0.5 * (T[k == 4, 0, 0] + T[k == 4, 0, 1]) + rng.normal(size=(np.sum(k == 4), 3)) * scale * 1e-5
    # a corner (5) or an edge (6) of A on B's plane or about the tolerance off it; 7: A's corner about there beside B
    m = k >= 5
    a, b, c = T[m, 1, 0], T[m, 1, 1], T[m, 1, 2]
    nn = np.cross(b - a, c - a)
    nn /= np.linalg.norm(nn, axis=1, keepdims=True)
    off = nn * (10.0 ** rng.uniform(-16, -4, size=(len(a), 1)) * rng.choice([-1, 0, 1], size=(len(a), 1)) * scale)
    w = rng.dirichlet((1, 1, 1), size=len(a))
    inside = w[:, :1] * a + w[:, 1:2] * b + w[:, 2:] * c
    T[m, 0, 0] = inside + off
    e = k[m] == 6
    T[np.nonzero(m)[0][e], 0, 1] = (0.3 * a + 0.7 * b + off)[e]
    s = k[m] == 7
    out = a + (b - a) * rng.uniform(0, 1, size=(len(a), 1))
    out += np.cross(b - a, nn) * 10.0 ** rng.uniform(-9, -2, size=(len(a), 1))
    T[np.nonzero(m)[0][s], 0, 0] = (out + off)[s]
    return T


@pytest.mark.parametrize("scale", [1e-4, 1e-3, 1.0, 100.0])
def test_parts_are_the_whole_and_planes_rule_out_no_segment(tmp_path, scale):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path / "tri_parts_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "zedm-x_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "tri_parts_check.cpp")], check=True, timeout=300)
    T = _pairs(np.random.default_rng(int(scale * 1e4)), 40000, scale)
    text = "\n".join(" ".join("%016x" % x for x in row) for row in T.reshape(len(T), 18).view(np.uint64))
    p = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=300)
    n, seg, out, differ, differ_np, wrong = (int(x) for x in p.stdout.split())
    assert n == len(T) and seg > 4000 and out > 4000
    assert (differ, differ_np, wrong) == (0, 0, 0)
