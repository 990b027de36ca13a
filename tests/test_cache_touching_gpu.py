"""The clearance cache where boxes touch without overlapping, with every margin the config key accepts: a lattice of
cubes whose faces coincide exactly (dyadic sizes and places, no rotation), first as laid out, then with every second
cube moved apart or into its neighbours by a few ulps to a few percent.  The box compares are strict, so triangles
whose boxes touch are tested; state and counters as without the cache, bit for bit."""
import numpy as np
import pytest

from _dem_helpers import box_tris, fmt, write_binary_stl, write_config

pytestmark = pytest.mark.gpu

H = 2.0 ** -10
SIDE = (7, 7, 6)  # 294 cubes: the cache is on from 256


def _scene(tmp_path, cache, tau):
    from zdemx.dem import Scene

    stl = str(tmp_path / "cube.stl")
    write_binary_stl(stl, box_tris(2 * H, 2 * H, 2 * H))
    parts = [dict(stl=stl, pos=fmt(2 * H * np.array(i)), vel="0 0 0", quat="1 0 0 0", omega="0 0 0", scale=1, density=2500,
                  young=1e7, poisson=0.25, mu=0.5, restitution=0.5)
             for i in np.ndindex(*SIDE)]
    cfg = str(tmp_path / f"c{cache}.txt")
    write_config(cfg, dict(steps=100, dt=1e-9, split_contacts=1, center_mesh=0, gravity="0 0 0", output_interval=1000,
                           output_dir=str(tmp_path / "out"), contact_cache=cache, contact_cache_tau=tau), parts)
    return Scene(cfg)


@pytest.mark.parametrize("tau", ["0", "-0.01", "nan", "0.005"])
def test_touching_boxes(tmp_path, tau):
    off, on = _scene(tmp_path, 0, tau), _scene(tmp_path, 1, tau)
    start = off.state()[0]
    odd = np.array([sum(i) % 2 for i in np.ndindex(*SIDE)], bool)
    touched = 0
    for shift in (0.0, 2.0 ** -60, -(2.0 ** -52), 2.0 ** -30, 0.01 * H, 0.0):
        st = start.copy()
        st[odd, 0] += shift
        for s in (off, on):
            s.set_state(st)
            s.step_graph(2)
        for x, y, name in zip(off.state(), on.state(), ("state", "force", "torque", "contact_count")):
            assert np.array_equal(x, y), (shift, name)
        a, b = off.info(), on.info()
        for k in ("contacts", "tri_checks", "segments", "comps", "loops", "pairs"):
            assert a[k] == b[k], (shift, k)
        touched += a["segments"] if shift == 0.0 else 0
    assert touched > 1000
