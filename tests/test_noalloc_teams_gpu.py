"""zdx_pair_contacts_noalloc's rebuild by teams, small slots and small lists: against the plain per-stage call (a warp a
pair), bit for bit, with pairs of every class, pairs that no class holds (a tolerance of half the body lists every two
segments), meshes of 20 triangles, and a triangle soup whose overlaps fill the lists many times over.  The device's
free memory stays what the first call left, whichever kernels a later call takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("ncontact", "contact_off", "stats", "geom", "info")


def _dev(lib, pm, pp):
    import torch

    meshes = {k: torch.from_numpy(np.ascontiguousarray(getattr(lib, k))).cuda() for k in ("tris", "tri_off", "mean_edge", "bbox_diag")}
    return meshes, {"mesh": torch.from_numpy(pm).cuda(), "pose": torch.from_numpy(pp).cuda()}


def _both(ctx, meshes, pairs, **kw):
    import torch

    from zdemx import _lib

    n, res = int(pairs["mesh"].shape[0]), []
    for call in (lambda o: _lib.pair_contacts_noalloc(ctx, meshes, pairs, o, k=1e7, **kw),
                 lambda o: _lib.pair_contacts_device(ctx, meshes, pairs, o, k=1e7, sched=_lib.SCHED_PER_STAGE, **kw)):
        out = {"ncontact": torch.zeros(n, dtype=torch.int32, device="cuda"), "stats": torch.zeros(n, 4, dtype=torch.int32, device="cuda"),
               "contact_off": torch.zeros(n + 1, dtype=torch.int64, device="cuda"),
               "geom": torch.zeros(8192, 20, dtype=torch.float64, device="cuda"),
               "info": torch.zeros(8192, 4, dtype=torch.int32, device="cuda")}
        torch.cuda.synchronize()
        before = ctx.timings()["launches"]
        tot = call(out)
        res.append((tot[:3], {k: v.cpu().numpy() for k, v in out.items()}, ctx.timings()["launches"] - before))
    (t0, a, launched), (t1, b, _) = res
    assert t0 == t1
    for k in KEYS:
        assert np.array_equal(a[k], b[k]), k
    return a, launched


@pytest.mark.parametrize("mode,split,tol", [(0, True, 0.0), (0, False, 0.0), (1, True, 1e-6)])
def test_every_class_and_the_rest(mode, split, tol):
    import torch

    from zdemx import _lib, synth
    from zdemx.contact import MeshLibrary

    rng = np.random.default_rng(21)
    lib = MeshLibrary.build([synth.noised_icosphere(s, 1e-3, 0.15, rng) for s in (0, 0, 1, 1, 2, 2, 4, 4)])
    pm, pp = [], []
    for m, n, depth in ((0, 40, 0.2), (2, 40, 0.2), (4, 30, 0.2), (6, 24, 0.15), (6, 12, 0.5)):
        pm += [(m, m + 1)] * n
        pp.append(synth.pair_poses(rng, n, 1e-3, 0.5 * depth, depth))
    pm, pp = np.array(pm, np.int32), np.concatenate(pp)
    ctx = _lib.Context(0)
    try:
        meshes, pairs = _dev(lib, pm, pp)
        some = {k: v[:80].contiguous() for k, v in pairs.items()}  # the first class alone
        a, small = _both(ctx, meshes, some, mode=mode, split=split, tol=tol)
        nseg = a["stats"][:, 0]
        assert nseg.max() <= 330
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        out = {"ncontact": torch.zeros(len(pm), dtype=torch.int32, device="cuda"),
               "stats": torch.zeros(len(pm), 4, dtype=torch.int32, device="cuda"),
               "contact_off": torch.zeros(len(pm) + 1, dtype=torch.int64, device="cuda"),
               "geom": torch.zeros(8192, 20, dtype=torch.float64, device="cuda"),
               "info": torch.zeros(8192, 4, dtype=torch.int32, device="cuda")}
        torch.cuda.synchronize()
        held = free - torch.cuda.mem_get_info()[0]  # torch's own
        _lib.pair_contacts_noalloc(ctx, meshes, pairs, out, k=1e7, mode=mode, split=split, tol=tol)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free - held
        a, all_ = _both(ctx, meshes, pairs, mode=mode, split=split, tol=tol)
        nseg = a["stats"][:, 0]
        for lo, hi in ((0, 330), (330, 560), (560, 1024)):
            assert np.any((nseg > lo) & (nseg <= hi)), (lo, hi, np.sort(nseg)[-20:])
        assert all_ == small + 2  # two classes more, and no pair went to the warps
    finally:
        ctx.close()


def test_pairs_that_no_class_holds():
    from zdemx import _lib, synth
    from zdemx.contact import MeshLibrary

    rng = np.random.default_rng(22)
    lib = MeshLibrary.build([synth.noised_icosphere(4, 1e-3, 0.15, rng) for _ in range(2)])
    pp = synth.pair_poses(rng, 6, 1e-3, 0.1, 0.15)
    ctx = _lib.Context(0)
    try:
        meshes, pairs = _dev(lib, np.tile(np.array([[0, 1]], np.int32), (6, 1)), pp)
        a, fine = _both(ctx, meshes, pairs, mode=1, split=True, tol=1e-6)
        assert a["stats"][:, 0].min() > 330
        b, coarse = _both(ctx, meshes, pairs, mode=1, split=True, tol=5e-4)
        assert coarse == fine + 1
    finally:
        ctx.close()


def test_small_meshes_and_full_lists():
    from zdemx import _lib, synth
    from zdemx.contact import MeshLibrary

    rng = np.random.default_rng(23)
    lib = MeshLibrary.build([synth.noised_icosphere(0, 1e-3, 0.15, rng) for _ in range(4)])
    n = 700
    pm = rng.integers(0, 4, size=(n, 2)).astype(np.int32)
    # deep enough that the boxes of most triangles meet: 20 x 20 pairs, lists of 120
    pp = synth.pair_poses(rng, n, 1e-3, 0.2, 1.6)
    ctx = _lib.Context(0)
    try:
        a, _ = _both(ctx, *_dev(lib, pm, pp), mode=0, split=True, tol=0.0)
        assert a["stats"][:, 0].max() > 20
        soup = MeshLibrary.build([rng.normal(size=(60, 3, 3)) * 1e-3 for _ in range(2)], center=False)
        pose = np.zeros((3, 14))
        pose[:, [3, 10]] = 1.0
        pose[1:, 7:10] = rng.normal(size=(2, 3)) * 2e-4
        a, _ = _both(ctx, *_dev(soup, np.tile(np.array([[0, 1]], np.int32), (3, 1)), pose), mode=0, split=False, tol=0.0)
        assert a["stats"][:, 0].max() > 500
    finally:
        ctx.close()
