"""Triangle pairs with slivers whose computed planes lean (test_plane_margin_cpu.py), one triangle a mesh, through the
batched call: segments and contacts as in the per-stage form, which has no plane test, and as in the oracle."""
import numpy as np
import pytest

from test_plane_margin_cpu import LOST, sliver_pairs

pytestmark = pytest.mark.gpu


def _call(ctx, T, pose, mode, sched):
    from zdemx import _lib

    n = len(T)
    off = np.arange(2 * n + 1, dtype=np.int64)
    edge = np.full(2 * n, 0.1)
    pm = np.arange(2 * n, dtype=np.int32).reshape(n, 2)
    return _lib.pair_contacts_raw(ctx, T.reshape(2 * n, 9), off, edge, edge, pm, pose, mode=mode, split=True, tol=1e-6, k=1.0,
                                  sched=sched)


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_slivers_keep_their_segments(ctx, mode):
    from zdemx import _lib

    rng = np.random.default_rng(17)
    T = np.concatenate([np.stack([LOST, LOST[::-1]])] + [sliver_pairs(rng, 6000, s) for s in (0.1, 1.0, 10.0)])
    pose = np.zeros((len(T), 14))
    pose[:, [3, 10]] = 1.0
    turn = rng.normal(size=(len(T), 4))
    pose[2:, 3:7] = pose[2:, 10:14] = (turn / np.linalg.norm(turn, axis=1, keepdims=True))[2:]
    new, old = (_call(ctx, T, pose, mode, s) for s in (_lib.SCHED_BATCHED, _lib.SCHED_PER_STAGE))
    assert np.array_equal(new["stats"][:, 0], old["stats"][:, 0]), np.nonzero(new["stats"][:, 0] != old["stats"][:, 0])[0]
    assert old["stats"][:, 0].sum() > 500
    for key in ("ncontact", "contact_off", "stats", "geom", "info"):
        assert np.array_equal(new[key], old[key]), key


def test_the_lost_pair_matches_the_oracle(ctx, oracle):
    from zdemx import _lib

    pose = np.zeros((1, 14))
    pose[:, [3, 10]] = 1.0
    for T in (LOST, LOST[::-1]):
        want = oracle.pair(T[0].reshape(1, 9), 0.1, 0.1, T[1].reshape(1, 9), pose[0, :7], pose[0, 7:], split=True, mode=0, tol=0.0)
        assert want["nseg"] == 1
        for sched in (_lib.SCHED_BATCHED, _lib.SCHED_PER_STAGE, _lib.SCHED_PLAIN):
            assert _call(ctx, T[None], pose, 0, sched)["stats"][0, 0] == 1, sched
