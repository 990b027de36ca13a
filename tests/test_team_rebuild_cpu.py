"""The team form of the rebuild (zdx_team.cuh), host build with a team of one, against the oracle: the same
components, loops and contacts, to the bit, in all three modes, for single pairs and for packs; every memory
size either gives that or refuses the pack without having written anything."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from _helpers import expected_contacts

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"
_dp, _ip, _lp = C.POINTER(C.c_double), C.POINTER(C.c_int), C.POINTER(C.c_longlong)


@pytest.fixture(scope="module")
def team(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("team") / "team.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CUDA_INC, "-I",
                    os.path.join(ROOT, "zedm-x_b200", "csrc"), "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "team_rebuild_check.cpp")], check=True, timeout=300)
    lib = C.CDLL(so)
    f = lib.team_rebuild_host
    f.argtypes = [C.c_int, _ip, _lp, _dp, _dp, _dp, _dp, C.c_int, C.c_int, C.c_double, C.c_double, C.c_int, C.c_int, _dp, _ip,
                  _dp, _ip, C.c_int, _ip, C.c_longlong, _lp, _lp]

    def call(pack, mode, split, tol, mem=1 << 22):
        """pack: (oracle result, mean edge, bbox diagonal, pose) of each pair."""
        segs = [np.asarray(r["seg"], float).reshape(-1, 6) for r, _, _, _ in pack]
        nseg = np.array([len(s) for s in segs], np.int32)
        off = np.r_[0, np.cumsum(nseg)].astype(np.int64)
        n, np_ = int(off[-1]), len(pack)
        cap = 4 * n + 64 * np_
        comp_cap = int(nseg.max()) + 1
        ar = {"seg": np.concatenate(segs), "me": np.array([x[1] for x in pack]), "bd": np.array([x[2] for x in pack]),
              "pose": np.array([x[3] for x in pack], float), "geom": np.zeros((cap, 20)),
              "info": np.zeros((cap, 4), np.int32), "points": np.zeros((cap, 3)),
              "comp": np.zeros((np_, comp_cap, 3), np.int32), "tape": np.zeros(64 * n + 4096, np.int32),
              "ctape": np.zeros(cap, np.int64), "pair": np.zeros((np_, 6), np.int64)}
        g = lambda k, t: ar[k].ctypes.data_as(t)
        ar["n"] = f(np_, nseg.ctypes.data_as(_ip), off.ctypes.data_as(_lp), g("seg", _dp), g("me", _dp), g("bd", _dp),
                    g("pose", _dp), mode, int(split), tol, 1e7, mem, cap, g("geom", _dp), g("info", _ip), g("points", _dp),
                    g("comp", _ip), comp_cap, g("tape", _ip), len(ar["tape"]), g("ctape", _lp), g("pair", _lp))
        return ar

    call.lib = lib
    return call


def _pairs(oracle, split, mode, tols):
    """Seeded pairs with segments, as the pack entries of `call` with a name: icospheres and hulls, of like
    and of very different sizes."""
    from zdemx import synth

    rng = np.random.default_rng(77)
    raw = []
    for la, lb in ((1, 1), (1, 2), (2, 2), (1, 3), (3, 1), (2, 3), (3, 3), (1, 4), (4, 2), (4, 4)):
        for _ in range(4 if max(la, lb) < 4 else 2):
            raw.append((synth.noised_icosphere(la, 1e-3, 0.15, rng), synth.noised_icosphere(lb, 1e-3, 0.15, rng),
                        synth.pair_poses(rng, 1, 1e-3, 0.05, 0.5)[0], f"ico {la} {lb}"))
    for _ in range(6):
        a, b = (synth.ellipsoid_hull(int(rng.integers(12, 200)), (1.0, 0.8, 0.6), 1e-3, rng) for _ in range(2))
        raw.append((a, b, synth.pair_poses(rng, 1, 1e-3, 0.6, 0.9)[0], "hull"))
    out = {t: [] for t in tols}
    for A, B, pose, name in raw:
        (A, pa), (B, _) = oracle.build_mesh(A, True), oracle.build_mesh(B, True)
        for tol in tols:
            r = oracle.pair(A, pa[5], pa[6], B, pose[:7], pose[7:], split=split, mode=mode, tol=tol)
            if r["nseg"]:
                out[tol].append((r, pa[5], pa[6], pose, f"{name} tol {tol}"))
    return out


def _check(o, k, entry, polyline):
    """Pair k of a pack's result against its oracle result."""
    r, name = entry[0], entry[4]
    e = expected_contacts(r, polyline=polyline)
    n, c0, npts, p0, ncomp, nloop = (int(x) for x in o["pair"][k])
    assert n == len(e["geom"]) and ncomp == r["ncomp"] and nloop == r["nloop"], name
    geom, info = o["geom"][c0: c0 + n], o["info"][c0: c0 + n]
    assert np.array_equal(geom[:, :13], e["geom"]), name
    assert np.array_equal(info[:, 0], np.full(n, k)) and np.array_equal(info[:, 1], np.arange(n)), name
    assert np.array_equal(info[:, 2], e["nvert"]) and np.array_equal(info[:, 3], e["comp"]), name
    pts = np.concatenate(e["points"]) if n else np.zeros((0, 3))
    assert npts == len(pts) and np.array_equal(o["points"][p0: p0 + npts], pts), name
    for c in range(ncomp):
        want = (r["comp_off"][c + 1] - r["comp_off"][c], r["v_off"][c + 1] - r["v_off"][c], r["e2_off"][c + 1] - r["e2_off"][c])
        assert tuple(o["comp"][k, c]) == want, name
    # tape: each contact's record holds its length and its vertices' endpoints
    seg = np.asarray(r["seg"]).reshape(-1, 6)
    for x in range(n):
        rec = o["tape"][o["ctape"][c0 + x]:]
        assert rec[0] == e["nvert"][x] and rec[1] == 0, name
        off = rec[1: 2 + rec[0]]
        mem = rec[2 + rec[0]: 2 + rec[0] + off[-1]]
        for q in range(rec[0]):
            m = mem[off[q]: off[q + 1]]
            s = np.zeros(3)
            for y in m:
                s = s + seg[y >> 1, 3 * (y & 1): 3 * (y & 1) + 3]
            assert np.array_equal(s / float(len(m)), e["points"][x][q]), name
    return n


MODES = [(0, True), (0, False), (1, True), (1, False), (2, True), (2, False)]


@pytest.mark.parametrize("mode,split", MODES)
def test_team_rebuild_matches_oracle(team, oracle, mode, split):
    seen = big = cut = most = 0
    for tol, entries in _pairs(oracle, split, mode, (0.0,) if mode == 0 else (1e-6, 2e-5)).items():
        for en in entries:
            o = team([en[:4]], mode, split, tol)
            if o["n"] == -1:  # more than 16 splits of one edge, or a neighbour test that is not symmetric
                cut += 1
                continue
            seen += _check(o, 0, en, mode != 0)
            big, most = max(big, en[0]["nseg"]), max(most, en[0]["ncomp"])
    assert seen > 40 and big > 300 and cut <= 2
    if split and mode:
        assert most > 16  # components sorted: above 16 std::sort and Python's sort part


@pytest.mark.parametrize("mode,split", MODES)
@pytest.mark.parametrize("size", [2, 5, 32])
def test_packs_match_oracle(team, oracle, mode, split, size):
    tol = 0.0 if mode == 0 else 2e-5
    entries = [e for e in _pairs(oracle, split, mode, (tol,))[tol] if e[0]["nseg"] <= 120]
    seen = 0
    for b in range(0, len(entries), size):
        pack = entries[b: b + size]
        o = team([e[:4] for e in pack], mode, split, tol)
        assert o["n"] >= 0
        seen += sum(_check(o, k, e, mode != 0) for k, e in enumerate(pack))
    assert seen > 20


def test_order_of_equal_keys(team):
    assert not any(team.lib.team_equal_order_differs(n) for n in range(3000))


def test_warp_sort_is_std_sort(team):
    """Also where introsort's depth runs out (many keys in adverse patterns)."""
    bad = [(n, keys, pattern, seed) for n in list(range(0, 70)) + [100, 127, 128, 129, 333, 1000, 2800]
           for keys in (1, 2, 3, 7, 300) for pattern in range(4) for seed in range(3)
           if team.lib.team_std_sort_differs(n, keys, pattern, seed)]
    assert not bad


def test_team_rebuild_memory_sizes(team, oracle):
    """From too little to plenty: refused, or the same result."""
    refused = held = 0
    entries = _pairs(oracle, True, 0, (0.0,))[0.0]
    for pack in [[e] for e in entries[::5]] + [entries[:3], entries[8:12]]:
        n = sum(e[0]["nseg"] for e in pack)
        for per in list(range(40, 400, 8)) + [500, 801]:
            o = team([e[:4] for e in pack], 0, True, 0.0, mem=per * n)
            assert o["n"] >= -1
            if o["n"] == -1:
                refused += 1
            else:
                held += 1
                for k, e in enumerate(pack):
                    _check(o, k, e, False)
    assert refused > 20 and held > 20
