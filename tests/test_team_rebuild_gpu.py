"""The team form of the rebuild on the GPU against the warp-per-pair form (which the plain per-stage schedule
runs): same contacts, loop points and per-pair counts, bit for bit, on batches that reach every class of
segment counts, the pairs above the last one and packs of the smallest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLASS_ENDS = (330, 560, 1150)  # largest segment counts of the classes of zdx_team.cu


def _batch():
    """Pairs of 1 to 1,800 segments, sizes mixed in every claim of a block."""
    from zdemx import synth
    from zdemx.contact import MeshLibrary

    rng = np.random.default_rng(31)
    levels = (0, 1, 2, 3, 4, 5)
    lib = MeshLibrary.build([synth.noised_icosphere(s, 1e-3, 0.15, rng) for s in levels for _ in range(2)])
    pm, pp = [], []
    for la, lb, n, depth in ((0, 0, 60, 0.2), (0, 1, 60, 0.2), (1, 1, 80, 0.1), (1, 2, 60, 0.1), (2, 2, 40, 0.2), (3, 3, 30, 0.2),
                             (1, 4, 12, 0.1), (4, 4, 24, 0.15), (4, 4, 16, 0.6), (5, 2, 6, 0.2), (5, 5, 4, 0.15)):
        for _ in range(n):
            pm.append((2 * la + rng.integers(0, 2), 2 * lb + rng.integers(0, 2)))
        pp.append(synth.pair_poses(rng, n, 1e-3, 0.5 * depth, depth))
    order = rng.permutation(len(pm))
    return lib, np.array(pm, np.int32)[order], np.concatenate(pp)[order]


@pytest.mark.parametrize("mode,split,tol", [(0, True, 0.0), (0, False, 0.0), (1, False, 1e-6), (1, True, 3e-5), (2, False, 2e-5),
                                            (2, True, 1e-6)])
def test_teams_match_warp_form(ctx, mode, split, tol):
    from zdemx import _lib

    lib, pm, pp = _batch()
    res = [_lib.pair_contacts_raw(ctx, lib.tris, lib.tri_off, lib.mean_edge, lib.bbox_diag, pm, pp, mode=mode, split=split,
                                  tol=tol, k=1e7, want_points=True, sched=s, comp_cap=64, point_cap=1 << 20)
           for s in (_lib.SCHED_BATCHED, _lib.SCHED_PER_STAGE)]
    for key in ("ncontact", "contact_off", "stats", "geom", "info", "points", "point_off", "comp_stats"):
        assert np.array_equal(res[0][key], res[1][key]), key
    n = res[0]["stats"][:, 0]
    assert res[0]["totals"][0] > 500
    ends = (0,) + CLASS_ENDS + (1 << 30,)
    for lo, hi in zip(ends[:-1], ends[1:]):
        assert np.any((n > lo) & (n <= hi)), (lo, hi, np.sort(n)[-40:])


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 150, 1000])
def test_small_and_odd_batches(ctx, n):
    """Blocks with one pair, with a few, and with a last claim that is not full."""
    from zdemx import _lib, synth
    from zdemx.contact import MeshLibrary, pair_contacts_batch

    rng = np.random.default_rng(n)
    lib = MeshLibrary.build([synth.noised_icosphere(s, 1e-3, 0.15, rng) for s in (1, 1, 2, 2, 3)])
    pm = rng.integers(0, lib.n_mesh, size=(n, 2)).astype(np.int32)
    pp = synth.pair_poses(rng, n, 1e-3, -0.1, 0.2)
    res = [pair_contacts_batch(ctx, lib, pm, pp, want_points=True, sched=s) for s in (_lib.SCHED_BATCHED, _lib.SCHED_PER_STAGE)]
    for key in ("ncontact", "contact_off", "stats", "geom", "info", "points", "point_off"):
        assert np.array_equal(res[0][key], res[1][key]), key
