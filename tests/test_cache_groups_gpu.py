"""The clearance cache's skip pass takes a warp's share of the pairs together, up to 16 consecutive ones (their motion
a lane each, then all their near pairs): scenes whose pairs give each warp one pair, a few, and all 16 with some
left over, against the same steps without the cache, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 4000, 33000])
def test_skip_pass_groups(tmp_path, n):
    from zdemx.dem import Scene
    from zdemx.workloads import pour_scene

    scenes = []
    for cache in (0, 1):
        cfg = pour_scene(str(tmp_path / f"c{cache}"), n=n, seed=7, steps=1000, vel_sigma=0.3)
        text = open(cfg).read().replace("split_contacts = 1", f"split_contacts = 1\ncontact_cache = {cache}")
        open(cfg, "w").write(text)
        scenes.append(Scene(cfg))
    off, on = scenes
    skipped = 0
    for chunk in (1, 2, 9):
        for s in scenes:
            s.step_graph(chunk)
        skipped += on.graph_cache()["skipped"]
        for x, y, name in zip(off.state(), on.state(), ("state", "force", "torque", "contact_count")):
            assert np.array_equal(x, y), f"{name} differs after {off.info()['steps']} steps"
        for k in ("contacts", "tri_checks", "segments", "comps", "loops", "pairs"):
            assert off.info()[k] == on.info()[k], k
    assert skipped > 0
