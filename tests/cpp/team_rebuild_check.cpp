// Host build of zdx_team.cuh (the rebuild of a pack of pairs by a team of threads) with a team of one, for
// tests/test_team_rebuild_cpu.py: a shared library.
#include <cstring>
#include <vector>

#include "zdx_team.cuh"

using namespace zdx;

// np pairs; pair k has nseg[k] segments from seg + 6 * seg_off[k], mean_edge[k], bbox_diag[k], pose + 14 k.
// Returns the number of contacts, -1 when the pack is not held in `bytes` of memory, -2 when a result moved
// all the same, -3 when memory behind them was written.  geom 20, info 4 a contact; per pair of pair_out:
// contacts, first contact, loop points, first loop point, components, raw loops.
extern "C" int team_rebuild_host(int np, const int* nseg, const long long* seg_off, const double* seg,
                                 const double* mean_edge, const double* bbox_diag, const double* pose, int mode, int split,
                                 double tol, double k, int bytes, int cap, double* geom, int* info, double* pts,
                                 int* comp_stats, int comp_cap, int* tape, long long tape_cap, long long* ctape,
                                 long long* pair_out) {
    PairArgs a{};
    std::vector<int32_t> pmesh(2 * np), ncon(np, -1), ncomp(np, -1), nloop(np, -1), status(np, 0), clen(cap);
    std::vector<int64_t> stage(np, -1), pstage(np, -1), npt(np, -1);
    unsigned long long cc = 0, pc = 0, tc = 0;
    int err = 0;
    for (int p = 0; p < np; ++p) pmesh[2 * p] = pmesh[2 * p + 1] = p;
    a.mean_edge = mean_edge;
    a.bbox_diag = bbox_diag;
    a.pmesh = pmesh.data();
    a.pose = pose;
    a.mode = mode;
    a.split = split;
    a.tol_in = tol;
    a.k = k;
    a.want_pts = pts ? 1 : 0;
    a.seg = const_cast<double*>(seg);
    a.pair_seg_off = reinterpret_cast<int64_t*>(const_cast<long long*>(seg_off));
    a.pair_nseg = const_cast<int*>(nseg);
    a.pair_status = status.data();
    a.cgeom_stage = geom;
    a.cinfo_stage = info;
    a.clen_stage = clen.data();
    a.contact_cap = cap;
    a.contact_counter = &cc;
    a.pts_stage = pts;
    a.pts_cap = cap;
    a.pts_counter = &pc;
    a.pair_stage_off = stage.data();
    a.pair_pts_stage_off = pstage.data();
    a.pair_ncontact = ncon.data();
    a.pair_npts = npt.data();
    a.pair_ncomp = ncomp.data();
    a.pair_nloop = nloop.data();
    a.err = &err;
    a.comp_stats = comp_stats;
    a.comp_stats_cap = comp_cap;
    a.tape_stage = tape;
    a.tape_cap = tape_cap;
    a.tape_counter = &tc;
    a.ctape_stage = reinterpret_cast<int64_t*>(ctape);
    TeamShared sh;
    std::memset(&sh, 0x5a, sizeof(sh));
    for (int p = 0; p < np; ++p) sh.pr[p].p = p;
    HostTeam tm;
    tm.sh = &sh;
    // exactly `bytes`, with a guard behind, so that a write past the end shows
    std::vector<double> mem((size_t)bytes / 8 + 16, 0.0);
    char* base = reinterpret_cast<char*>(mem.data());
    std::memset(base, 0x5a, mem.size() * 8);
    const bool ok = mode == 2 ? team_rebuild<HostTeam, true>(tm, a, np, base, bytes)
                              : team_rebuild<HostTeam, false>(tm, a, np, base, bytes);
    for (size_t i = (size_t)bytes; i < mem.size() * 8; ++i)
        if (base[i] != 0x5a) return -3;
    if (!ok) {
        for (int p = 0; p < np; ++p)
            if (ncon[p] != -1) return -2;
        return cc || pc || tc || err ? -2 : -1;
    }
    if (err) return -4;
    for (int p = 0; p < np; ++p) {
        const long long o[6] = {ncon[p], stage[p], npt[p], pstage[p], ncomp[p], nloop[p]};
        std::memcpy(pair_out + 6 * p, o, sizeof(o));
    }
    return (int)cc;
}

// Where team_equal_sorted puts n equal keys, and where the std::sort restatement does.
extern "C" int team_equal_order_differs(int n) {
    std::vector<int> idx(n), got(n, -1);
    for (int i = 0; i < n; ++i) idx[i] = i;
    std_sort_idx(idx.data(), n, [](int, int) { return false; });
    for (int i = 0; i < n; ++i) got[team_equal_sorted(i, n)] = i;
    return got == idx ? 0 : 1;
}

// team_std_sort of n words with keys below `keys`, against the std::sort restatement; pattern 0 random, 1 mostly
// key 0, 2 ascending runs, 3 descending.
extern "C" int team_std_sort_differs(int n, int keys, int pattern, unsigned seed) {
    std::vector<int> a(n);
    unsigned s = seed * 2654435761u + 1u;
    auto next = [&]() { return (s = s * 1664525u + 1013904223u) >> 8; };
    for (int i = 0; i < n; ++i) {
        const int k = pattern == 0   ? (int)(next() % keys)
                      : pattern == 1 ? (next() % 8 == 0 ? (int)(next() % keys) : 0)
                      : pattern == 2 ? i % keys
                                     : keys - 1 - (int)((long long)i * keys / n);
        a[i] = k << 16 | i;
    }
    std::vector<int> b = a;
    std::vector<unsigned short> l(n + 1), r(n + 1), leaf(n + 1);
    HostTeam tm;
    std_sort_idx(a.data(), n, [](int x, int y) { return (x >> 16) < (y >> 16); });
    team_std_sort(tm, b.data(), n, l.data(), r.data(), leaf.data());
    return a == b ? 0 : 1;
}
