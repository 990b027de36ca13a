"""The adjoint's warp takes a loop's vertices 32 at a time and their endpoints 32 at a time: loops below,
around and above these strides (icospheres of 80, 1280 and 5120 triangles) against central differences.

The step is h = 1e-6 R, the edges are at least R / 20 long: truncation leaves (20 h / R)^2 = 4e-10 of the
gradient's scale, rounding 1e-16 / 1e-6 = 1e-10 of it times the spread of the vertices' shares (below 1e3),
so 1e-6 holds for both.
"""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fd():
    spec = importlib.util.spec_from_file_location(
        "adjoint_fd", os.path.join(os.path.dirname(os.path.abspath(__file__)), "test_adjoint_gpu.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("level", [1, 3, 4])
def test_adjoint_long_loops(ctx, level):
    from zdemx import synth
    from zdemx.contact import MeshLibrary

    fd = _fd()
    rng = np.random.default_rng(40 + level)
    lib = MeshLibrary.build([synth.noised_icosphere(level, fd.R, 0.1, rng) for _ in range(2)])
    pose = synth.pair_poses(rng, 2, fd.R, 0.06, 0.12)
    pose[:, 3:7] = synth.random_unit_quat(rng, 2)
    fd._fd_check(ctx, lib, pose, np.array([[0, 1], [1, 0]], np.int32), mode=0, split=True, tol=0.0, rng=rng)
