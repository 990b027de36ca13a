"""The team form of the rebuild holds the pairs it is meant to: a pair that no class holds goes to the warp-per-pair
kernel, one launch more, so the number of launches says whether any did.  (test_team_rebuild_gpu.py compares the two
forms; a class that held nothing would compare the warp form with itself.)"""
import numpy as np
import pytest

from test_team_rebuild_gpu import CLASS_ENDS, _batch

pytestmark = pytest.mark.gpu


def _call(ctx, lib, pm, pp, mode, split, tol):
    from zdemx import _lib

    before = ctx.timings()["launches"]
    r = _lib.pair_contacts_raw(ctx, lib.tris, lib.tri_off, lib.mean_edge, lib.bbox_diag, pm, pp, mode=mode, split=split, tol=tol,
                               k=1e7, want_points=True, contact_cap=1 << 16, point_cap=1 << 21)
    return r, ctx.timings()["launches"] - before


@pytest.mark.parametrize("mode,split,tol", [(0, True, 0.0), (0, False, 0.0), (1, False, 1e-6), (1, True, 3e-5), (2, False, 2e-5),
                                            (2, True, 1e-6)])
def test_every_class_holds_its_pairs(ctx, mode, split, tol):
    lib, pm, pp = _batch()
    n = _call(ctx, lib, pm, pp, mode, split, tol)[0]["stats"][:, 0]
    # pairs without segments are settled where the classes are made: no class is launched, and nothing can be refused
    apart = pp.copy()
    apart[:, 7:10] += 1.0
    r, base = _call(ctx, lib, pm, apart, mode, split, tol)
    assert r["stats"][:, 0].max() == 0
    for c, (lo, hi) in enumerate(zip((0,) + CLASS_ENDS[:-1], CLASS_ENDS)):
        sel = np.nonzero((n > lo) & (n <= hi))[0]
        assert len(sel) >= 12
        # together, in packs, and the largest of the class alone
        for some in (sel, sel[np.argsort(-n[sel])][:1]):
            assert _call(ctx, lib, pm[some], pp[some], mode, split, tol)[1] == base + 1 + c, (lo, hi, len(some))
    sel = np.nonzero(n <= CLASS_ENDS[-1])[0]
    assert _call(ctx, lib, pm[sel], pp[sel], mode, split, tol)[1] == base + len(CLASS_ENDS)
    # and above the last class the warp form is launched
    over = np.nonzero(n > CLASS_ENDS[-1])[0][:1]
    assert _call(ctx, lib, pm[over], pp[over], mode, split, tol)[1] == base + len(CLASS_ENDS) + 1
