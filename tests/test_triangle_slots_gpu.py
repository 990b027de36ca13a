"""The triangle stage's slots: what a context holds after a large batch of small meshes, and a batch with a pair whose
segments outgrow the smaller slots of many CTAs (it runs again with whole ones): same results as the pair alone, and
the per-pair limit as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_workspace_of_a_large_batch_of_small_meshes():
    """Two whole slots an SM (16,384 segments of 58 bytes and the survivors) and 256 MB for everything else."""
    import torch

    from zdemx import _lib, synth
    from zdemx.contact import MeshLibrary, pair_contacts_batch

    rng = np.random.default_rng(3)
    lib = MeshLibrary.build([synth.noised_icosphere(2, 1e-3, 0.15, rng) for _ in range(4)])
    n = 3000
    pm = rng.integers(0, lib.n_mesh, size=(n, 2)).astype(np.int32)
    pp = synth.pair_poses(rng, n, 1e-3, 0.0, 0.1)
    ctx = _lib.Context(0)
    try:
        pair_contacts_batch(ctx, lib, pm[:64], pp[:64])  # the module and its code are loaded
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        pair_contacts_batch(ctx, lib, pm, pp)
        torch.cuda.synchronize()
        held = free - torch.cuda.mem_get_info()[0]
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert held < 2 * sms * 16384 * 58 + (256 << 20), held
        # a count that climbs past every number of CTAs takes no more
        free = torch.cuda.mem_get_info()[0]
        for m in (310, 460, 880, 900, 2999):
            pair_contacts_batch(ctx, lib, pm[:m], pp[:m])
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] >= free
    finally:
        ctx.close()


def _soup(rng, n, size):
    """n triangles thrown across a ball: most cut many of another soup's."""
    return rng.normal(size=(n, 3, 3)) * size


@pytest.mark.parametrize("limit", [0, 7000, 1500])
def test_a_pair_that_outgrows_its_slot(limit):
    import ctypes as C

    from zdemx import _lib, synth

    rng = np.random.default_rng(8)
    small = [synth.noised_icosphere(1, 1e-3, 0.15, rng) for _ in range(4)]
    meshes = small + [_soup(rng, 180, 1e-3) for _ in range(2)]
    off = np.concatenate([[0], np.cumsum([len(m) for m in meshes])]).astype(np.int64)
    tris = np.concatenate(meshes).reshape(-1, 9)
    edge, diag = np.full(len(meshes), 1e-4), np.full(len(meshes), 2e-3)
    n = 1200
    pm = rng.integers(0, len(small), size=(n, 2)).astype(np.int32)
    pp = synth.pair_poses(rng, n, 1e-3, 0.0, 0.1)
    pm[700] = (4, 5)
    pp[700] = 0.0
    pp[700, [3, 10]] = 1.0

    def call(ctx, sel):
        m, p = np.ascontiguousarray(pm[sel]), np.ascontiguousarray(pp[sel])
        k, cap = len(m), 40 * len(m) + 4096
        out = {"ncontact": np.zeros(k, np.int32), "contact_off": np.zeros(k + 1, np.int64), "stats": np.zeros((k, 4), np.int32),
               "geom": np.zeros((cap, 20)), "info": np.zeros((cap, 4), np.int32)}
        ptr = lambda x: x.ctypes.data
        opts = _lib.PairOpts(0, 0, 0.0, 1.0, _lib.MEM_HOST, _lib.SCHED_BATCHED, 0, limit)
        ms = _lib.MeshSet(len(meshes), ptr(tris), ptr(off), ptr(edge), ptr(diag))
        res = _lib.PairResult(ptr(out["ncontact"]), ptr(out["contact_off"]), ptr(out["stats"]), cap, ptr(out["geom"]),
                              ptr(out["info"]), 0, 0, 0)
        rc = _lib.lib().zdx_pair_contacts(ctx.handle, C.byref(opts), C.byref(ms), C.byref(_lib.PairBatch(k, ptr(m), ptr(p))),
                                          C.byref(res))
        return rc, out

    ctx = _lib.Context(0)
    try:
        rc1, alone = call(ctx, np.array([700]))
        results = [call(ctx, np.arange(n)) for _ in range(2)]  # with the rerun, and with what it taught the context
    finally:
        ctx.close()
    nseg = int(alone["stats"][0, 0])
    if limit:
        assert nseg == limit and rc1 != 0 and alone["stats"][0, 3] & 1
    else:
        assert 6000 < nseg < 16384 and rc1 == 0  # 888 CTAs' slots hold about 5,400
    for rc, out in results:
        assert rc == rc1
        assert np.array_equal(out["stats"][700], alone["stats"][0])
        if rc == 0:
            a, b = out["contact_off"][700], out["contact_off"][701]
            assert b - a == alone["contact_off"][1] and b > a
            assert np.array_equal(out["geom"][a:b], alone["geom"][: b - a])
            assert np.array_equal(out["info"][a:b, 1:], alone["info"][: b - a, 1:])
    assert all(np.array_equal(results[0][1][k], results[1][1][k]) for k in alone)
