// zdx_team.cuh -- the rebuild stage of a pack of pairs by a team of threads, with all of the pairs' arrays in one
// block of (shared) memory.
//
// Same results as rebuild_pair in zdx_pair.cu, bit for bit (both follow src/main.cpp:2148-2219 and
// polyline.py:743-829).  What the reference does one segment, endpoint or edge at a time is laid out as
// passes over flat lists of the whole pack (its pairs' segments one after the other), so that the lanes are
// full and few passes wait on a chain of dependent loads:
//   * box tests of all segment pairs (32 x 32 tiles, outward-rounded floats) list the few that overlap;
//     lanes over that list take the cell ranks, the endpoint distances and the segment distances;
//   * components by a lock-free union-find over the accepted pairs.  The search order inside a component
//     (src/main.cpp:874-897) is then a depth-first walk over sorted neighbour lists, a warp a
//     component, its lanes over the list of the segment popped;
//   * the snap is a union-find over the endpoints of listed pairs (two endpoints within h lie in adjacent
//     cells, so their segments are listed); links point at the smaller endpoint, so a class's root is its
//     first appearance and vertex ids are a scan;
//   * T-junctions: lanes over edges list the vertices in reach, lanes over that list test them;
//   * loops: one thread a component walks them; lanes over all loop vertices compute the terms of Sn and
//     Gn, and one thread per sum adds them in loop order.
// A pack that a pass cannot hold (memory, index range, a neighbour test that is not symmetric, more than 16
// splits of one edge) makes the function return false before anything is written outside `sm`.
//
// The code is written against a Team (thread index, size, barrier, scan, atomics), so that it also runs on
// the host with a team of one.
#pragma once
#include <cmath>
#include <cstdint>

#include "zdx_math.cuh"
#include "zdx_npmath.cuh"
#include "zdx_pair.cuh"
#include "zdx_pyset.cuh"
#include "zdx_sortrep.cuh"

namespace zdx {

// Pairs of a pack, and the segments it may have: the lists keep segment indices in 13 bits.
constexpr int TEAM_PACK = 32;
constexpr int TEAM_MAX_SEG = 4096;

struct TeamPair {
    int p, n;
    int comp0, loop0;  // its first component and raw loop in the pack
    double h, area_eps;
    V3 dirAB;
    I3 c0;  // cell of its first point
};
// What a team shares beside the arrays: the pack (p of each pair is the caller's), counters, partial sums.
struct TeamShared {
    TeamPair pr[TEAM_PACK];
    int first[TEAM_PACK + 1];  // first segment of each pair
    int n_list, n_near, bad, hits;
    int part[32];
    unsigned long long cbase, pbase, tbase;
    int np, from, to, claimed[TEAM_PACK];  // the kernel's: pairs of this pack, the items it has claimed
};

#if defined(__CUDACC__)
// T threads: one warp, or the whole block.
template <int T_>
struct DevTeam {
    static constexpr int T = T_;
    static constexpr int LANES = 32, WARPS = T / 32;
    int t;
    TeamShared* sh;
    __device__ __forceinline__ int lane() const { return t & 31; }
    __device__ __forceinline__ int warp() const { return t >> 5; }
    __device__ __forceinline__ unsigned below() const { return (1u << (t & 31)) - 1u; }
    static __device__ __forceinline__ void warp_sync() { __syncwarp(); }
    static __device__ __forceinline__ unsigned ballot(bool b) { return __ballot_sync(0xffffffffu, b); }
    static __device__ __forceinline__ int from_lane(int v, int l) { return __shfl_sync(0xffffffffu, v, l); }
    static __device__ __forceinline__ int popc(unsigned b) { return __popc(b); }
    static __device__ __forceinline__ int last(unsigned b) { return 31 - __clz(b); }
    __device__ __forceinline__ void sync() const {
        if constexpr (T == 32) __syncwarp();
        else __syncthreads();
    }
    // exclusive prefix of v over the team; *total receives the sum
    __device__ __forceinline__ int scan(int v, int* total) const {
        const int lane = t & 31;
        int x = v;
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if constexpr (T == 32) {
            *total = __shfl_sync(0xffffffffu, x, 31);
            return x - v;
        } else {
            if (lane == 31) sh->part[t >> 5] = x;
            __syncthreads();
            int before = 0, all = 0;
            for (int w = 0; w < T / 32; ++w) {
                const int s = sh->part[w];
                if (w < (t >> 5)) before += s;
                all += s;
            }
            __syncthreads();
            *total = all;
            return before + x - v;
        }
    }
    static __device__ __forceinline__ int add(int* p, int v) { return atomicAdd(p, v); }
    static __device__ __forceinline__ int cas(int* p, int was, int v) { return atomicCAS(p, was, v); }
    static __device__ __forceinline__ void max(int* p, int v) { atomicMax(p, v); }
    static __device__ __forceinline__ unsigned long long take(unsigned long long* p, unsigned long long v) {
        return atomicAdd(p, v);
    }
    static __device__ __forceinline__ void flag(int* p, int v) { atomicOr(p, v); }
};
#endif

// A team of one, on the host.
struct HostTeam {
    static constexpr int T = 1;
    static constexpr int LANES = 1, WARPS = 1;
    int t = 0;
    TeamShared* sh = nullptr;
    ZDX_HD int lane() const { return 0; }
    ZDX_HD int warp() const { return 0; }
    ZDX_HD unsigned below() const { return 0u; }
    static ZDX_HD void warp_sync() {}
    static ZDX_HD unsigned ballot(bool b) { return b ? 1u : 0u; }
    static ZDX_HD int from_lane(int v, int) { return v; }
    static ZDX_HD int popc(unsigned b) { return (int)(b & 1u); }
    static ZDX_HD int last(unsigned) { return 0; }
    ZDX_HD void sync() const {}
    ZDX_HD int scan(int v, int* total) const {
        *total = v;
        return 0;
    }
    static ZDX_HD int add(int* p, int v) {
        const int o = *p;
        *p += v;
        return o;
    }
    static ZDX_HD void max(int* p, int v) { *p = *p < v ? v : *p; }
    static ZDX_HD int cas(int* p, int was, int v) {
        const int o = *p;
        if (o == was) *p = v;
        return o;
    }
    static ZDX_HD unsigned long long take(unsigned long long* p, unsigned long long v) {
        const unsigned long long o = *p;
        *p += v;
        return o;
    }
    static ZDX_HD void flag(int* p, int v) { *p |= v; }
};

// Bump allocation in [lo, hi) of the pair's memory, in 16-byte steps.  Every thread computes the same
// offsets; ok turns false once the room is exceeded, before anything is written there.
struct TeamMem {
    char* base;
    int lo, hi;
    bool ok;
    ZDX_HD char* bytes(long n) {
        const long o = ((long)lo + n + 15) & ~15L;
        char* p = base + lo;
        if (o > hi) ok = false;
        else lo = (int)o;
        return p;
    }
    template <class X>
    ZDX_HD X* take(long n) {
        return reinterpret_cast<X*>(bytes((long)sizeof(X) * n));
    }
    ZDX_HD bool fits(long n) const { return (((long)lo + n + 15) & ~15L) <= hi; }
};

ZDX_HD float team_down(double x) {
#if defined(__CUDA_ARCH__)
    return __double2float_rd(x);
#else
    const float f = (float)x;
    return (double)f > x ? std::nextafterf(f, -INFINITY) : f;
#endif
}
ZDX_HD float team_up(double x) {
#if defined(__CUDA_ARCH__)
    return __double2float_ru(x);
#else
    const float f = (float)x;
    return (double)f < x ? std::nextafterf(f, INFINITY) : f;
#endif
}
ZDX_HD V3 team_ld(const double* p) { return V3{p[0], p[1], p[2]}; }
ZDX_HD void team_st(double* p, V3 v) {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
}
// Cells are kept relative to the pair's first one in 16 bits; a pair that spans more is not held here.
ZDX_HD bool team_cell(I3 c, I3 c0, I3* out) {
    const long long x = (long long)c.x - c0.x, y = (long long)c.y - c0.y, z = (long long)c.z - c0.z;
    const long long m = 16000;
    *out = I3{(int)x, (int)y, (int)z};
    return x >= -m && x <= m && y >= -m && y <= m && z >= -m && z <= m;
}
ZDX_HD void team_put(short* p, I3 c) {
    p[0] = (short)c.x;
    p[1] = (short)c.y;
    p[2] = (short)c.z;
    p[3] = 0;
}
ZDX_HD I3 team_get(const short* p) {
#if defined(__CUDA_ARCH__)
    const short4 v = *reinterpret_cast<const short4*>(p);
    return I3{v.x, v.y, v.z};
#else
    return I3{p[0], p[1], p[2]};
#endif
}
ZDX_HD bool team_adjacent(I3 a, I3 b) {
    const int dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return !(dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1);
}

// Union-find whose links point at smaller indices, so that a root is its class's smallest member.  A link
// is made by a compare-and-swap on a root; losing the race means it is no root any more.
ZDX_HD int team_root(const volatile int* par, int x) {
    int p = par[x];
    while (p != x) {
        x = p;
        p = par[x];
    }
    return x;
}
// The root of x, shortening the way there: every other node is hung under its grandparent (an ancestor in the
// same class whatever other threads do meanwhile; roots are changed by the swap below alone).
ZDX_HD int team_root_halving(volatile int* par, int x) {
    int p = par[x];
    while (p != x) {
        const int g = par[p];
        if (g == p) return p;
        par[x] = g;
        x = g;
        p = par[x];
    }
    return x;
}
template <class Team>
ZDX_HD void team_unite(int* par, int a, int b) {
    for (;;) {
        a = team_root_halving(par, a);
        b = team_root_halving(par, b);
        if (a == b) return;
        if (a > b) {
            const int s = a;
            a = b;
            b = s;
        }
        if (Team::cas(par + b, b, a) == b) return;
    }
}

// Where std::sort leaves element x of n equal ones: up to 16 in place (insertion); else the median of three
// equal keys swaps the first with the middle, the partition reverses the rest, and both parts follow.
ZDX_HD int team_equal_sorted(int x, int n) {
    int f = 0, l = n;
    while (l - f > 16) {
        const int mid = f + (l - f) / 2;
        if (x == f) x = mid;
        else if (x == mid) x = f;
        if (x > f) x = f + l - x;
        const int cut = f + 1 + (l - f - 1) / 2;
        if (x < cut) l = cut;
        else f = cut;
    }
    return x;
}

// std::sort (std_sort_idx) of n packed words, key in the upper 16 bits, by one warp: the same permutation.  A
// Hoare partition swaps the k-th word from the left that is not below the pivot with the k-th from the right
// that is not above it, as long as the first lies left of the second, so the two lists (built here by
// ballots, in left / right) give every swap at once.  Where the k-th two have crossed, the scan from the left
// stops at its k-th word or at the last one swapped to the right, whichever comes first: the cut.  What
// the partitions leave (ranges of 16 at most, every word of one not above any of the next) is sorted by a
// lane a range: an insertion sort is stable, so the one over everything moves no word out of its range.
template <class Team>
ZDX_HD void team_std_sort(const Team& tm, int* f, int n, unsigned short* left, unsigned short* right,
                          unsigned short* leaf) {
    const int lane = tm.lane();
    auto key = [&](int i) { return f[i] >> 16; };
    int lg = 0;
    while ((1 << (lg + 1)) <= n) lg++;
    int lo_stack[34], hi_depth[34];  // first | last << 16, depth: every lane has the same
    int sp = 0, leaves = 0;
    lo_stack[0] = n << 16;
    hi_depth[0] = 2 * lg;
    sp = 1;
    while (sp > 0) {
        --sp;
        const int first = lo_stack[sp] & 0xffff;
        int last = (int)((unsigned)lo_stack[sp] >> 16), depth = hi_depth[sp];
        while (last - first > 16) {
            if (depth == 0) {
                if (lane == 0) sr_heapsort(f + first, last - first, [](int x, int y) { return (x >> 16) < (y >> 16); });
                break;
            }
            --depth;
            // median of first + 1, middle, last - 1 to the front
            const int b = first + (last - first) / 2;
            const int ka = key(first + 1), kb = key(b), kc = key(last - 1);
            const int m = ka < kb ? (kb < kc ? b : ka < kc ? last - 1 : first + 1) : ka < kc ? first + 1 : kb < kc ? last - 1 : b;
            tm.warp_sync();
            if (lane == 0) {
                const int w = f[first];
                f[first] = f[m];
                f[m] = w;
            }
            tm.warp_sync();
            const int pivot = key(first);
            int nl = 0, nr = 0;
            for (int x = 0; x < last - first - 1; x += Team::LANES) {
                const int i = first + 1 + x + lane, j = last - 1 - x - lane;
                const bool l = i < last && key(i) >= pivot, r = j > first && key(j) <= pivot;
                const unsigned bl = tm.ballot(l), br = tm.ballot(r);
                if (l) left[nl + tm.popc(bl & tm.below())] = (unsigned short)i;
                if (r) right[nr + tm.popc(br & tm.below())] = (unsigned short)j;
                nl += tm.popc(bl);
                nr += tm.popc(br);
            }
            // the front itself stops the scan from the right, and some word not below the pivot the other
            if (lane == 0) {
                right[nr] = (unsigned short)first;
                left[nl] = (unsigned short)last;
            }
            tm.warp_sync();
            int cut = last;
            for (int k0 = 0;; k0 += Team::LANES) {
                const int k = k0 + lane;
                const bool in = k <= nl && k <= nr;
                const int i = in ? left[k] : 0, j = in ? right[k] : 0;
                const bool swap = in && i < j;
                if (swap) {
                    const int w = f[i];
                    f[i] = f[j];
                    f[j] = w;
                }
                const unsigned stop = tm.ballot(!swap);
                if (stop) {
                    const int before = in && k > 0 ? right[k - 1] : last;
                    cut = tm.from_lane(i < before ? i : before, Team::popc((stop & (0u - stop)) - 1u));
                    break;
                }
            }
            tm.warp_sync();
            lo_stack[sp] = cut | last << 16;
            hi_depth[sp++] = depth;
            last = cut;
        }
        if (lane == 0) leaf[leaves] = (unsigned short)first;
        ++leaves;
    }
    tm.warp_sync();
    // the ranges were met left to right (one that ran out of depth is sorted already)
    for (int x = lane; x < leaves; x += Team::LANES) {
        const int e0 = leaf[x], e1 = x + 1 < leaves ? leaf[x + 1] : n;
        for (int i = e0 + 1; i < e1; ++i) {
            const int w = f[i];
            int y = i - 1;
            while (y >= e0 && (w >> 16) < key(y)) {
                f[y + 1] = f[y];
                --y;
            }
            f[y + 1] = w;
        }
    }
    tm.warp_sync();
}

// In-place exclusive scan of v[0..n) into v[0..n], v[n] = total.
template <class Team>
ZDX_HD int team_scan(const Team& tm, int* v, int n) {
    int run = 0;
    for (int b = 0; b < n; b += Team::T) {
        const int i = b + tm.t;
        const int x = i < n ? v[i] : 0;
        int tot;
        const int ex = tm.scan(x, &tot);
        if (i < n) v[i] = run + ex;
        run += tot;
    }
    if (tm.t == 0) v[n] = run;
    tm.sync();
    return run;
}

template <bool NPX>
ZDX_HD bool team_close(V3 a, V3 b, double h, bool py) {
    const V3 d = a - b;
    if constexpr (NPX) return np::norm3(&d.x) <= h;
    return py ? (sqrt(dot(d, d)) <= h) : (dot(d, d) <= h * h);
}

// The part of a loop's contact that follows from its two sums (src/main.cpp:1042-1052, 2188-2219;
// polyline.py:211-218): |Sn|, nA, xc0, and whether the loop is a contact.  `diag` is polyline mode's
// bounding-box diagonal.
template <bool NPX>
ZDX_HD bool team_contact(V3 Sn, V3 Gn, double diag, bool py, double tol, double area_eps, V3 dirAB, double& area, V3& nA,
                         V3& xc0) {
    if constexpr (NPX) area = np::norm3(&Sn.x);
    else area = norm(Sn);
    nA = V3{0.0, 0.0, 0.0};
    xc0 = V3{0.0, 0.0, 0.0};
    if (!py) {
        if (area < 1e-14) return false;
        nA = Sn * (-1.0 / area);
        xc0 = cross(nA, Gn) / area;
        if (area < area_eps) return false;
        if (dot(nA, dirAB) < 0.0) nA = nA * -1.0;
        return true;
    }
    if (diag < tol * 2) return false;
    if (area < 1e-14) {
        area = 0.0;
    } else {
        nA = V3{-Sn.x / area, -Sn.y / area, -Sn.z / area};
        xc0 = cross(nA, Gn) / area;
    }
    return true;
}

// The rebuild of the pairs sh.pr[0..np), each with at least one segment and status 0.  False: the pack is not
// held here (see above).
template <class Team, bool NPX>
ZDX_HD bool team_rebuild(const Team& tm, const PairArgs& a, const int np, char* sm, const int bytes) {
    TeamShared& sh = *tm.sh;
    const bool py = NPX || a.mode == 1;
    const bool split = a.split != 0;
    // polyline.py's search visits a segment's candidates, all those with adjacent rep cells, in the order of a
    // Python set (zdx_pyset.cuh)
    const bool by_set = py && split;
    // Lanes that leave an item early wait for the others of their warp: left to themselves they go on to their
    // next items apart (the trip count is the same for every lane, so that all of them get to the wait).
    auto each = [&](int count, auto&& f) {
        for (int b = 0; b < count; b += Team::T) {
            if (b + tm.t < count) f(b + tm.t);
            tm.warp_sync();
        }
    };
    each(np, [&](int k) {
        TeamPair& P = sh.pr[k];
        const int p = P.p;
        const int mA = a.pmesh[2 * (int64_t)p];
        const double* ps = a.pose + 14 * (int64_t)p;
        const double me = a.mean_edge[mA];
        double tol = a.tol_in;
        if (!(tol > 0.0)) {
            tol = me > 0.0 ? (me * 0.1) : (a.bbox_diag[mA] * 1e-2);
            if (tol <= 0.0) tol = 1e-6;
        }
        P.n = a.pair_nseg[p];
        P.h = tol;
        P.area_eps = me > 0.0 ? (me * me * 1e-4) : 1e-12;
        P.dirAB = V3{ps[7], ps[8], ps[9]} - V3{ps[0], ps[1], ps[2]};
        P.c0 = cell_of(team_ld(a.seg + 6 * a.pair_seg_off[p]), tol);
    });
    tm.sync();
    if (tm.t == 0) {
        int run = 0;
        for (int k = 0; k < np; ++k) {
            sh.first[k] = run;
            run = run > TEAM_MAX_SEG ? run : run + sh.pr[k].n;
        }
        sh.first[np] = run;
        sh.n_list = sh.n_near = sh.bad = sh.hits = 0;
    }
    tm.sync();
    const int n = sh.first[np];
    if (n > TEAM_MAX_SEG) return false;

    TeamMem M{sm, 0, bytes & ~15, true};
    double* S = M.take<double>(6L * n);
    short* rc = M.take<short>(12L * n);  // rep cells (p0, p1, mid), relative to the pair's c0
    const int low_end = M.lo;            // dead once the vertices are known
    unsigned short* ord = M.take<unsigned short>(n);  // segments in component order
    unsigned short* pos = M.take<unsigned short>(n);  // and back
    unsigned short* cc = M.take<unsigned short>(n);   // component of a segment
    unsigned short* comp_off = M.take<unsigned short>(n + 1);
    unsigned char* sp = M.take<unsigned char>(n);  // pair of a segment
    unsigned char* cp = M.take<unsigned char>(n);  // pair of a component
    if (!M.ok || !M.fits(32L * n)) return false;

    // ---- segments, rep cells, padded boxes (src/main.cpp:815-833)
    M.hi -= 32 * n;
    float4* bx = reinterpret_cast<float4*>(sm + M.hi);  // min x y z, max x | max y, max z
    each(n, [&](int i) {
        int k = 0, d = np;  // first[k] <= i < first[d]
        while (d - k > 1) {
            const int m = (k + d) >> 1;
            if (sh.first[m] <= i) k = m;
            else d = m;
        }
        sp[i] = (unsigned char)k;
        const TeamPair& P = sh.pr[k];
        const double h = P.h;
        // boxes that overlap wherever rep cells are adjacent, for which the set wants all
        const double hb = by_set ? h * (1.0 + 1e-6) : h;
        const double* g = a.seg + 6 * (a.pair_seg_off[P.p] + (i - sh.first[k]));
        const V3 p0 = team_ld(g), p1 = team_ld(g + 3);
        team_st(S + 6 * i, p0);
        team_st(S + 6 * i + 3, p1);
        bool in = true;
        for (int r = 0; r < 3; ++r) {
            I3 c;
            in = team_cell(cell_of(r == 0 ? p0 : r == 1 ? p1 : (p0 + p1) * 0.5, h), P.c0, &c) && in;
            team_put(rc + 12 * i + 4 * r, c);
        }
        bx[2 * i] = float4{team_down(smin(p0.x, p1.x) - hb), team_down(smin(p0.y, p1.y) - hb), team_down(smin(p0.z, p1.z) - hb),
                           team_up(smax(p0.x, p1.x) + hb)};
        bx[2 * i + 1] = float4{team_up(smax(p0.y, p1.y) + hb), team_up(smax(p0.z, p1.z) + hb), 0.f, 0.f};
        if (!in) sh.bad = 1;
    });
    tm.sync();

    // ---- every two segments i < j of a pair whose boxes overlap: tiles of 32 i (a lane each) by 32 j (read by
    // all lanes at once; a j of its own for every lane waits on the banks instead)
    uint32_t* list = reinterpret_cast<uint32_t*>(sm + M.lo);
    const int list_cap = (M.hi - M.lo) / 4;
    {
        int k = 0, ti = 0, first = 0, nt = (sh.pr[0].n + 31) >> 5;  // pair, tile row, the row's first task
        for (int q = tm.t;; q += Team::T) {
            const int task = q >> 5;
            while (k < np && task - first >= nt - ti) {
                first += nt - ti;
                if (++ti == nt) {
                    ti = 0;
                    if (++k < np) nt = (sh.pr[k].n + 31) >> 5;
                }
            }
            if (k == np) break;
            const int b = sh.first[k], e = sh.first[k + 1];
            const int i = b + 32 * ti + (q & 31), j0 = b + 32 * (ti + task - first), j1 = j0 + 32 < e ? j0 + 32 : e;
            const float4 p0 = bx[2 * (i < e ? i : e - 1)], p1 = bx[2 * (i < e ? i : e - 1) + 1];
            // four at a time, their hits afterwards: the loads of one do not wait for the list of another
            for (int j = j0; j < j1; j += 4) {
                unsigned hit = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
                for (int r = 0; r < 4; ++r) {
                    const float4 o0 = bx[2 * (j + r < j1 ? j + r : j)], o1 = bx[2 * (j + r < j1 ? j + r : j) + 1];
                    // all six compares at once: a chain of short-circuits waits out a load for each
                    const bool apart = (p0.w < o0.x) | (p0.x > o0.w) | (p1.x < o0.y) | (p0.y > o1.x) | (p1.y < o0.z) | (p0.z > o1.y);
                    hit |= (!apart & (i < j + r) & (j + r < j1) & (i < e)) ? 1u << r : 0u;
                }
                for (int r = 0; hit; hit >>= 1, ++r) {
                    if (!(hit & 1u)) continue;
                    const int o = Team::add(&sh.n_list, 1);
                    if (o < list_cap) list[o] = (uint32_t)i | (uint32_t)(j + r) << 16;
                }
                tm.warp_sync();  // or the lanes go on apart, each with its own rest of the tile
            }
        }
    }
    tm.sync();
    const int nlist = sh.n_list;
    if (sh.bad || nlist > list_cap) return false;
    M.hi = bytes & ~15;  // the boxes are dead

    // ---- the neighbours among them: some rep cells adjacent.  Entry: i | j << 13 | walk rank of j from i
    // << 26 | of i from j << 33 | close endpoints (bit 2 ei + ej) << 40 | DFS edge << 44 | boxes meet << 45.  They grow down
    // from the end of the memory.
    unsigned long long* near_top = reinterpret_cast<unsigned long long*>(sm + M.hi);
    const int near_cap = (M.hi - ((M.lo + 4 * nlist + 15) & ~15)) / 8;
    each(nlist, [&](int k) {
        const int i = (int)(list[k] & 0xffffu), j = (int)(list[k] >> 16);
        const double h = sh.pr[sp[i]].h;
        const V3 a0 = team_ld(S + 6 * i), a1 = team_ld(S + 6 * i + 3), b0 = team_ld(S + 6 * j), b1 = team_ld(S + 6 * j + 3);
        // the reference's box test in FP64 (the floats only rule out)
        const bool meet =
            !(smax(a0.x, a1.x) + h < smin(b0.x, b1.x) - h || smin(a0.x, a1.x) - h > smax(b0.x, b1.x) + h ||
              smax(a0.y, a1.y) + h < smin(b0.y, b1.y) - h || smin(a0.y, a1.y) - h > smax(b0.y, b1.y) + h ||
              smax(a0.z, a1.z) + h < smin(b0.z, b1.z) - h || smin(a0.z, a1.z) - h > smax(b0.z, b1.z) + h);
        if (!meet && !by_set) return;
        // smallest walk rank r * 27 + cell over the adjacent rep points, from either side
        int kij = 127, kji = 127, close = 0;
        for (int r = 0; r < 3; ++r) {
            const I3 ci = team_get(rc + 12 * i + 4 * r);
            for (int s = 0; s < 3; ++s) {
                const I3 cj = team_get(rc + 12 * j + 4 * s);
                const int dx = cj.x - ci.x, dy = cj.y - ci.y, dz = cj.z - ci.z;
                if (dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1) continue;
                const int cell = (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1);
                const int k1 = r * 27 + cell, k2 = s * 27 + (26 - cell);
                kij = k1 < kij ? k1 : kij;
                kji = k2 < kji ? k2 : kji;
                if (r < 2 && s < 2 && team_close<NPX>(r ? a1 : a0, s ? b1 : b0, h, py)) close |= 1 << (2 * r + s);
            }
        }
        if (kij == 127 || (!split && !close)) return;
        const int o = Team::add(&sh.n_near, 1);
        if (o < near_cap)
            near_top[-1 - o] = (unsigned long long)i | (unsigned long long)j << 13 | (unsigned long long)kij << 26 |
                               (unsigned long long)kji << 33 | (unsigned long long)close << 40 |
                               (meet ? 1ull << 45 : 0ull);
    });
    tm.sync();
    const int nnear = sh.n_near;
    if (nnear > near_cap) return false;
    M.hi = (M.hi - 8 * nnear) & ~15;

    // ---- components and their order (label_segments_by_contact_greedy, src/main.cpp:804-898)
    int ncomp = np;
    if (split) {
        const int mark = M.lo;
        int* lab = M.take<int>(n);
        int* end = M.take<int>(n + 1);  // neighbour lists: counts, then ends
        unsigned short* root = M.take<unsigned short>(n);
        unsigned short* cid = M.take<unsigned short>(n);
        unsigned short* seed = M.take<unsigned short>(n);
        unsigned short* stack = M.take<unsigned short>(n);
        unsigned char* seen = M.take<unsigned char>(n);
        int* csort = M.take<int>(n + 1);
        if (!M.ok) return false;
        each(n, [&](int i) {
            lab[i] = i;
            end[i] = 0;
            seen[i] = 0;
            csort[i] = 0;
        });
        tm.sync();
        each(nnear, [&](int k) {
            const unsigned long long w = near_top[-1 - k];
            const int i = (int)(w & 0x1fff), j = (int)((w >> 13) & 0x1fff);
            const V3 a0 = team_ld(S + 6 * i), a1 = team_ld(S + 6 * i + 3), b0 = team_ld(S + 6 * j), b1 = team_ld(S + 6 * j + 3);
            const double tol2 = sh.pr[sp[i]].h * sh.pr[sp[i]].h;
            bool edge = false;
            if (w >> 45 & 1) {
                bool ij, ji;
                if constexpr (NPX) {
                    ij = np::seg_seg_dist2(&a0.x, &a1.x, &b0.x, &b1.x) <= tol2;
                    ji = np::seg_seg_dist2(&b0.x, &b1.x, &a0.x, &a1.x) <= tol2;
                } else {
                    ij = seg_seg_dist2(a0, a1, b0, b1) <= tol2;
                    ji = seg_seg_dist2(b0, b1, a0, a1) <= tol2;
                }
                // the search takes whichever direction it meets first: only where both agree is the component
                // known without it
                if (ij != ji) sh.bad = 1;
                edge = ij;
            }
            if (edge) {
                near_top[-1 - k] = w | 1ull << 44;
                team_unite<Team>(lab, i, j);
            }
            if (edge || by_set) {
                Team::add(end + i, 1);
                Team::add(end + j, 1);
            }
        });
        tm.sync();
        if (sh.bad) return false;
        each(n, [&](int i) { root[i] = (unsigned short)team_root(lab, i); });
        const int nadj = team_scan(tm, end, n);
        // components are found in the order of their smallest segment
        int found = 0;
        for (int b = 0; b < n; b += Team::T) {
            const int i = b + tm.t;
            const bool f = i < n && root[i] == i;
            int tot;
            const int ex = tm.scan(f ? 1 : 0, &tot);
            if (f) {
                cid[i] = (unsigned short)(found + ex);
                seed[found + ex] = (unsigned short)i;
            }
            found += tot;
        }
        ncomp = found;
        uint32_t* adj = M.take<uint32_t>(nadj);
        if (!M.ok || nadj > 0xffff) return false;
        tm.sync();
        each(nnear, [&](int k) {
            const unsigned long long w = near_top[-1 - k];
            const uint32_t edge = (uint32_t)(w >> 44 & 1);
            if (!edge && !by_set) return;
            const int i = (int)(w & 0x1fff), j = (int)((w >> 13) & 0x1fff);
            // walk rank << 16 | segment << 1 | DFS edge
            adj[Team::add(end + i, 1)] = (uint32_t)(w >> 26 & 0x7f) << 16 | (uint32_t)j << 1 | edge;
            adj[Team::add(end + j, 1)] = (uint32_t)(w >> 33 & 0x7f) << 16 | (uint32_t)i << 1 | edge;
        });
        each(n, [&](int i) { Team::add(csort + cid[root[i]], 1); });
        tm.sync();
        each(n, [&](int i) {
            const int e0 = i ? end[i - 1] : 0, e1 = end[i];
            for (int x = e0 + 1; x < e1; ++x) {
                const uint32_t v = adj[x];
                int y = x - 1;
                while (y >= e0 && adj[y] > v) {
                    adj[y + 1] = adj[y];
                    --y;
                }
                adj[y + 1] = v;
            }
            lab[i] = e0 | (e1 - e0) << 16;  // from here the segment's list: first entry, length
        });
        tm.sync();
        if (by_set) {
            // each list's edges alone, in the order of the set its candidates make when they are added in list order
            if (tm.t == 0) sh.hits = 0;
            tm.sync();
            each(n, [&](int i) { Team::max(&sh.hits, (int)((uint32_t)lab[i] >> 16)); });
            tm.sync();
            const int most = sh.hits, words = 10 * most + 8;
            const int left = (M.hi - M.lo) / 4 / words, lanes = left < Team::T ? left : Team::T;
            tm.sync();
            if (tm.t == 0) sh.hits = 0;
            if (lanes < 1) return false;
            int* tab = reinterpret_cast<int*>(sm + M.lo) + tm.t * words;
            for (int b = 0; b < n; b += lanes) {
                const int i = b + tm.t;
                if (tm.t < lanes && i < n) {
                    const int e0 = lab[i] & 0xffff, nc = (int)((uint32_t)lab[i] >> 16), s0 = sh.first[sp[i]];
                    int *old = tab + 8 * most + 8, *keys = old + most;
                    for (int q = 0; q < nc; ++q) keys[q] = ((int)(adj[e0 + q] & 0xffffu) >> 1) - s0;
                    bool ok = true;
                    const unsigned mask = pyset_build(keys, nc, tab, old, &ok);
                    if (!ok) sh.bad = 1;
                    int cnt = 0;
                    for (unsigned x = 0; x <= mask; ++x) {
                        if (tab[x] < 0) continue;
                        int q = 0;
                        while (keys[q] != tab[x]) ++q;
                        if (adj[e0 + q] & 1u) old[cnt++] = tab[x];
                    }
                    for (int q = 0; q < cnt; ++q) adj[e0 + q] = (uint32_t)(old[q] + s0) << 1 | 1u;
                    lab[i] = e0 | cnt << 16;
                }
                tm.warp_sync();
            }
            tm.sync();
            if (sh.bad) return false;
        }
        // a pair's components by size, descending, ties as std::sort leaves them (src/main.cpp:897; Python's sort is
        // stable), on packed words
        unsigned short* tmp = M.take<unsigned short>(3L * (ncomp + np));
        if (!M.ok) return false;
        for (int k = tm.warp(); k < np; k += Team::WARPS) {
            const int c0 = cid[sh.first[k]], c1 = k + 1 < np ? cid[sh.first[k + 1]] : ncomp;
            for (int c = c0 + tm.lane(); c < c1; c += Team::LANES) csort[c] = (32767 - csort[c]) << 16 | c;
            tm.warp_sync();
            unsigned short* t = tmp + 3 * (c0 + k);
            if (!py) team_std_sort(tm, csort + c0, c1 - c0, t, t + (c1 - c0) + 1, t + 2 * (c1 - c0) + 2);
            if (tm.lane() != 0) continue;
            if (py) stable_sort_idx(csort + c0, c1 - c0, [](int x, int y) { return (x >> 16) < (y >> 16); });
            sh.pr[k].comp0 = c0;
            int run = sh.first[k];
            for (int c = c0; c < c1; ++c) {
                comp_off[c] = (unsigned short)run;
                cp[c] = (unsigned char)k;
                run += 32767 - (csort[c] >> 16);
            }
        }
        if (tm.t == 0) comp_off[ncomp] = (unsigned short)n;
        tm.sync();
        // each component's search by a warp, lanes over the popped segment's list: what was not seen yet is pushed
        // in list order, so the last of it is popped next
        for (int k = tm.warp(); k < ncomp; k += Team::WARPS) {
            const int base = comp_off[k], size = comp_off[k + 1] - base;
            int i = seed[csort[k] & 0xffff], cnt = 1, sp_n = 0;
            if (tm.lane() == 0) {
                seen[i] = 1;
                ord[base] = (unsigned short)i;
                cc[i] = (unsigned short)k;
                pos[i] = (unsigned short)base;
            }
            while (cnt < size) {
                tm.warp_sync();
                int top = -1;
                const int e0 = lab[i] & 0xffff, e1 = e0 + (int)((uint32_t)lab[i] >> 16);
                for (int x0 = e0; x0 < e1; x0 += Team::LANES) {
                    const int x = x0 + tm.lane();
                    const int j = x < e1 ? (int)(adj[x] & 0xffffu) >> 1 : 0;
                    const bool fresh = x < e1 && !seen[j];
                    const unsigned bal = tm.ballot(fresh);
                    if (!bal) continue;
                    const int at = Team::popc(bal & tm.below()), lastl = Team::last(bal);
                    if (top >= 0 && tm.lane() == 0) stack[base + sp_n] = (unsigned short)top;
                    sp_n += top >= 0 ? 1 : 0;
                    if (fresh) {
                        seen[j] = 1;
                        ord[base + cnt + at] = (unsigned short)j;
                        cc[j] = (unsigned short)k;
                        pos[j] = (unsigned short)(base + cnt + at);
                        if (tm.lane() != lastl) stack[base + sp_n + at] = (unsigned short)j;
                    }
                    const int nb = Team::popc(bal);
                    top = tm.from_lane(j, lastl);
                    sp_n += nb - 1;
                    cnt += nb;
                }
                if (top < 0) {
                    tm.warp_sync();
                    top = stack[base + --sp_n];
                }
                i = top;
            }
        }
        tm.sync();
        M.lo = mark;
    } else {
        each(n, [&](int i) {
            ord[i] = pos[i] = (unsigned short)i;
            cc[i] = sp[i];
        });
        each(np + 1, [&](int k) {
            comp_off[k] = (unsigned short)sh.first[k];
            if (k == np) return;
            cp[k] = (unsigned char)k;
            sh.pr[k].comp0 = k;
        });
        tm.sync();
    }

    // ---- snap_endpoints (src/main.cpp:680-746) of all components: endpoint q = 2 position + end
    unsigned short* vq = M.take<unsigned short>(2L * n);
    int* vbase = M.take<int>(ncomp + 1);
    M.hi -= 8 * n;
    if (!M.ok || M.hi < M.lo) return false;
    int* par = reinterpret_cast<int*>(sm + M.hi);
    each(2 * n, [&](int q) { par[q] = q; });
    tm.sync();
    each(n, [&](int i) {
        if (team_adjacent(team_get(rc + 12 * i), team_get(rc + 12 * i + 4)) &&
            team_close<NPX>(team_ld(S + 6 * i + 3), team_ld(S + 6 * i), sh.pr[sp[i]].h, py))
            team_unite<Team>(par, 2 * pos[i], 2 * pos[i] + 1);
    });
    each(nnear, [&](int k) {
        const unsigned long long w = near_top[-1 - k];
        const int close = (int)(w >> 40 & 0xf);
        const int i = (int)(w & 0x1fff), j = (int)((w >> 13) & 0x1fff);
        if (!close || cc[i] != cc[j]) return;
        for (int c = 0; c < 4; ++c)
            if (close >> c & 1) team_unite<Team>(par, 2 * pos[i] + (c >> 1), 2 * pos[j] + (c & 1));
    });
    tm.sync();
    each(2 * n, [&](int q) { vq[q] = (unsigned short)team_root(par, q); });
    tm.sync();
    int nvt = 0;
    for (int b = 0; b < 2 * n; b += Team::T) {
        const int q = b + tm.t;
        const bool f = q < 2 * n && vq[q] == q;
        int tot;
        const int ex = tm.scan(f ? 1 : 0, &tot);
        if (f) par[q] = nvt + ex;
        nvt += tot;
    }
    tm.sync();
    each(2 * n, [&](int q) { vq[q] = (unsigned short)par[vq[q]]; });
    tm.sync();
    each(ncomp, [&](int c) { vbase[c] = vq[2 * comp_off[c]]; });
    if (tm.t == 0) vbase[ncomp] = nvt;
    M.hi = bytes & ~15;  // the neighbours and the links are dead
    double* V = M.take<double>(3L * nvt);
    short* vc = M.take<short>(4L * nvt);
    int* vend = M.take<int>(nvt + 1);  // a vertex's endpoints: counts, then ends in vmem
    unsigned short* vmem = M.take<unsigned short>(2L * n);
    const int after = M.lo;
    unsigned short* vany = M.take<unsigned short>(2L * n);  // in any order; dead once vmem is there
    if (!M.ok) return false;
    M.lo = after;
    each(nvt, [&](int v) { vend[v] = 0; });
    tm.sync();
    each(2 * n, [&](int q) { Team::add(vend + vq[q], 1); });
    tm.sync();
    team_scan(tm, vend, nvt);
    each(2 * n, [&](int q) { vany[Team::add(vend + vq[q], 1)] = (unsigned short)q; });
    tm.sync();
    // a vertex's endpoints in endpoint order, each to its rank (a tolerance above the segments' length joins
    // hundreds into one vertex)
    each(2 * n, [&](int x) {
        const int q = vany[x], v = vq[q];
        const int e0 = v ? vend[v - 1] : 0, e1 = vend[v];
        int r = e0;
        for (int y = e0; y < e1; ++y) r += vany[y] < q ? 1 : 0;
        vmem[r] = (unsigned short)q;
    });
    tm.sync();
    // each vertex: the mean of its endpoints, summed in that order
    each(nvt, [&](int v) {
        const int e0 = v ? vend[v - 1] : 0, e1 = vend[v];
        V3 s = team_ld(S + 6 * ord[vmem[e0] >> 1] + 3 * (vmem[e0] & 1));
        for (int x = e0 + 1; x < e1; ++x) s = s + team_ld(S + 6 * ord[vmem[x] >> 1] + 3 * (vmem[x] & 1));
        const V3 m = s / (double)(e1 - e0);
        team_st(V + 3 * v, m);
        const TeamPair& P = sh.pr[sp[ord[vmem[e0] >> 1]]];
        I3 c;
        if (!team_cell(cell_of(m, P.h), P.c0, &c)) sh.bad = 1;
        team_put(vc + 4 * v, c);
    });
    tm.sync();
    if (sh.bad) return false;

    // ---- edges in segment order; from here arrays go first where the segments and rep cells were
    TeamMem L{sm, 0, low_end, true};
    auto room = [&](long b) -> char* { return L.fits(b) ? L.bytes(b) : M.bytes(b); };
    uint32_t* E = reinterpret_cast<uint32_t*>(room(4L * n));
    unsigned short* ec = reinterpret_cast<unsigned short*>(room(2L * n));
    int* ebase = reinterpret_cast<int*>(room(4L * (ncomp + 1)));
    if (!M.ok) return false;
    int ne = 0;
    for (int b = 0; b < n; b += Team::T) {
        const int q = b + tm.t;
        const int va = q < n ? vq[2 * q] : 0, vb = q < n ? vq[2 * q + 1] : 0;
        const int f = va != vb ? 1 : 0;
        int tot;
        const int ex = tm.scan(f, &tot);
        if (q < n) {
            const int c = cc[ord[q]];
            if (q == comp_off[c]) ebase[c] = ne + ex;
            if (f) {
                E[ne + ex] = (uint32_t)va | (uint32_t)vb << 16;
                ec[ne + ex] = (unsigned short)c;
            }
        }
        ne += tot;
    }
    if (tm.t == 0) ebase[ncomp] = ne;
    int* eh = reinterpret_cast<int*>(room(4L * (ne + 1)));  // splits of an edge: counts, then ends
    if (!M.ok) return false;
    each(ne, [&](int e) { eh[e] = 0; });
    tm.sync();

    // ---- split_t_junctions (src/main.cpp:900-961): the vertices in an edge's cells, then the exact test
    if (tm.t == 0) sh.n_list = 0;
    tm.sync();
    uint32_t* tj = reinterpret_cast<uint32_t*>(sm + M.lo);
    const int tj_cap = (M.hi - M.lo) / 4;
    each(ne, [&](int e) {
        const int va = (int)(E[e] & 0xffffu), vb = (int)(E[e] >> 16);
        const V3 pa = team_ld(V + 3 * va), pb = team_ld(V + 3 * vb);
        const TeamPair& P = sh.pr[cp[ec[e]]];
        const double h = P.h;
        const V3 mn{smin(pa.x, pb.x) - h, smin(pa.y, pb.y) - h, smin(pa.z, pb.z) - h};
        const V3 mx{smax(pa.x, pb.x) + h, smax(pa.y, pb.y) + h, smax(pa.z, pb.z) + h};
        I3 lo, hi;
        if (!team_cell(cell_of(mn, h), P.c0, &lo) || !team_cell(cell_of(mx, h), P.c0, &hi)) {
            sh.bad = 1;
            return;
        }
        const int v1 = vbase[ec[e] + 1];
        for (int v = vbase[ec[e]]; v < v1; ++v) {
            const I3 c = team_get(vc + 4 * v);
            if ((c.x < lo.x) | (c.x > hi.x) | (c.y < lo.y) | (c.y > hi.y) | (c.z < lo.z) | (c.z > hi.z) | (v == va) | (v == vb))
                continue;
            const int k = Team::add(&sh.n_list, 1);
            if (k < tj_cap) tj[k] = (uint32_t)e << 16 | (uint32_t)v;
        }
    });
    tm.sync();
    const int ntj = sh.n_list;
    if (sh.bad || ntj > tj_cap) return false;
    auto edge_t = [&](int e, int v, double* t) {
        const double* pa = V + 3 * (E[e] & 0xffffu);
        const double* pb = V + 3 * (E[e] >> 16);
        if constexpr (NPX) return np::point_seg_dist2_t(V + 3 * v, pa, pb, t);
        return pt_seg_d2t(team_ld(V + 3 * v), team_ld(pa), team_ld(pb), *t);
    };
    each(ntj, [&](int k) {
        double t = 0.0;
        const double d2 = edge_t((int)(tj[k] >> 16), (int)(tj[k] & 0xffffu), &t);
        const double h = sh.pr[cp[ec[tj[k] >> 16]]].h;
        if (!(d2 <= h * h && t > 1e-6 && t < 1.0 - 1e-6)) {
            tj[k] = 0xffffffffu;
            return;
        }
        Team::add(eh + (tj[k] >> 16), 1);
        Team::add(&sh.hits, 1);
    });
    tm.sync();
    const int hits = sh.hits;
    uint32_t* E2 = E;
    int* ebase2 = ebase;
    int ne2 = ne;
    if (hits > 0) {
        M.bytes(4L * ntj);  // the list stays
        unsigned short* hv = reinterpret_cast<unsigned short*>(room(2L * hits));
        double* ht = reinterpret_cast<double*>(room(8L * hits));
        int* eo = reinterpret_cast<int*>(room(4L * (ne + 1)));
        ebase2 = reinterpret_cast<int*>(room(4L * (ncomp + 1)));
        if (!M.ok) return false;
        team_scan(tm, eh, ne);
        each(ntj, [&](int k) {
            if (tj[k] != 0xffffffffu) hv[Team::add(eh + (tj[k] >> 16), 1)] = (unsigned short)(tj[k] & 0xffffu);
        });
        tm.sync();
        // an edge's splits in the order of the reference's walk over cells (vertex id inside a cell), then
        // sorted by t: up to 16 of them std::sort is an insertion sort, which is stable
        each(ne, [&](int e) {
            const int e0 = e ? eh[e - 1] : 0, e1 = eh[e];
            if (e1 - e0 > 16) sh.bad = 1;
            for (int x = e0 + 1; x < e1; ++x) {
                const unsigned short v = hv[x];
                const I3 cv = team_get(vc + 4 * v);
                int y = x - 1;
                while (y >= e0) {
                    const I3 cy = team_get(vc + 4 * hv[y]);
                    const bool after = cy.x != cv.x   ? cy.x > cv.x
                                       : cy.y != cv.y ? cy.y > cv.y
                                       : cy.z != cv.z ? cy.z > cv.z
                                                      : hv[y] > v;
                    if (!after) break;
                    hv[y + 1] = hv[y];
                    --y;
                }
                hv[y + 1] = v;
            }
            for (int x = e0; x < e1; ++x) {
                const unsigned short v = hv[x];
                double t = 0.0;
                edge_t(e, v, &t);
                int y = x - 1;
                while (y >= e0 && t < ht[y]) {
                    hv[y + 1] = hv[y];
                    ht[y + 1] = ht[y];
                    --y;
                }
                hv[y + 1] = v;
                ht[y + 1] = t;
            }
            int prev = (int)(E[e] & 0xffffu), last = -1, cnt = 0;
            for (int x = e0; x <= e1; ++x) {
                const int v = x < e1 ? hv[x] : (int)(E[e] >> 16);
                if (x < e1 && v == last) continue;
                if (prev != v) ++cnt;
                prev = v;
                last = v;
            }
            eo[e] = cnt;
        });
        tm.sync();
        if (sh.bad) return false;
        ne2 = team_scan(tm, eo, ne);
        E2 = reinterpret_cast<uint32_t*>(room(4L * ne2));
        if (!M.ok) return false;
        each(ne, [&](int e) {
            const int e0 = e ? eh[e - 1] : 0, e1 = eh[e];
            int prev = (int)(E[e] & 0xffffu), last = -1, o = eo[e];
            for (int x = e0; x <= e1; ++x) {
                const int v = x < e1 ? hv[x] : (int)(E[e] >> 16);
                if (x < e1 && v == last) continue;
                if (prev != v) E2[o++] = (uint32_t)prev | (uint32_t)v << 16;
                prev = v;
                last = v;
            }
        });
        each(ncomp + 1, [&](int c) { ebase2[c] = eo[ebase[c]]; });
        tm.sync();
        // more edges than the warp-per-pair kernel holds
        each(np, [&](int k) {
            const int c1 = k + 1 < np ? sh.pr[k + 1].comp0 : ncomp;
            if (ebase2[c1] - ebase2[sh.pr[k].comp0] > 4 * sh.pr[k].n + 64) sh.bad = 1;
        });
        tm.sync();
        if (sh.bad) return false;
    }

    // ---- extract_loops (src/main.cpp:963-1025): edges of a vertex in edge order, start vertices by degree
    int* vdeg = reinterpret_cast<int*>(room(4L * (nvt + 1)));  // counts, then ends
    uint32_t* ve = reinterpret_cast<uint32_t*>(room(8L * ne2));  // edge << 16 | other vertex
    int* vord = reinterpret_cast<int*>(room(4L * nvt));
    unsigned long long* vtwo = reinterpret_cast<unsigned long long*>(room(8L * nvt));  // both edges of a vertex of two
    int* codd = reinterpret_cast<int*>(room(4L * ncomp));  // a component with other vertices
    unsigned short* stmp = reinterpret_cast<unsigned short*>(room(6L * (nvt + ncomp)));  // the sort's
    unsigned char* used = reinterpret_cast<unsigned char*>(room(ne2));
    unsigned short* lv = reinterpret_cast<unsigned short*>(room(2L * (ne2 + ncomp)));  // loop vertices
    unsigned short* le = reinterpret_cast<unsigned short*>(room(2L * (ne2 + 1)));      // a component's loop ends
    int* nl = reinterpret_cast<int*>(room(4L * (ncomp + 1)));
    if (!M.ok) return false;
    each(nvt, [&](int v) { vdeg[v] = 0; });
    each(ne2, [&](int e) { used[e] = 0; });
    each(ncomp, [&](int c) { codd[c] = 0; });
    tm.sync();
    each(ne2, [&](int e) {
        Team::add(vdeg + (E2[e] & 0xffffu), 1);
        Team::add(vdeg + (E2[e] >> 16), 1);
    });
    tm.sync();
    each(2 * n, [&](int q) {
        if (vdeg[vq[q]] != 2) codd[cc[ord[q >> 1]]] = 1;
    });
    tm.sync();
    // a vertex's sort key: two edges first, then by degree, descending (src/main.cpp:977-982).  Where every
    // vertex has two, the sorted place of each is known; the others are sorted below.
    each(nvt, [&](int v) {
        int c = 0, d = ncomp;  // vbase[c] <= v < vbase[d]
        while (d - c > 1) {
            const int m = (c + d) >> 1;
            if (vbase[m] <= v) c = m;
            else d = m;
        }
        if (codd[c]) vord[v] = (vdeg[v] == 2 ? 0 : 0x7fff - vdeg[v]) << 16 | v;
        else vord[py ? v : vbase[c] + team_equal_sorted(v - vbase[c], vbase[c + 1] - vbase[c])] = v;
    });
    tm.sync();
    team_scan(tm, vdeg, nvt);
    each(ne2, [&](int e) {
        const uint32_t x = E2[e] & 0xffffu, y = E2[e] >> 16;
        ve[Team::add(vdeg + x, 1)] = (uint32_t)e << 16 | y;
        ve[Team::add(vdeg + y, 1)] = (uint32_t)e << 16 | x;
    });
    tm.sync();
    each(nvt, [&](int v) {
        const int e0 = v ? vdeg[v - 1] : 0, e1 = vdeg[v];
        for (int x = e0 + 1; x < e1; ++x) {
            const uint32_t w = ve[x];
            int y = x - 1;
            while (y >= e0 && ve[y] > w) {
                ve[y + 1] = ve[y];
                --y;
            }
            ve[y + 1] = w;
        }
        vtwo[v] = e1 - e0 == 2 ? (unsigned long long)ve[e0 + 1] << 32 | ve[e0] : ~0ull;
    });
    tm.sync();
    if (!py) {
        for (int c = tm.warp(); c < ncomp; c += Team::WARPS) {
            const int v0 = vbase[c], nv = vbase[c + 1] - v0;
            if (!codd[c] || nv <= 16) continue;
            unsigned short* t = stmp + 3 * (v0 + c);
            team_std_sort(tm, vord + v0, nv, t, t + nv + 1, t + 2 * nv + 2);
        }
        tm.sync();
    }
    // one thread a component, neighbours in different warps (lanes that walk apart take turns)
    for (int c = tm.warp() + Team::WARPS * tm.lane(); c < ncomp; c += Team::T) {
        int* vo = vord + vbase[c];
        const int nv = vbase[c + 1] - vbase[c];
        // (up to 16 std::sort is an insertion sort, which is stable; more are sorted already)
        if (codd[c] && (py || nv <= 16)) stable_sort_idx(vo, nv, [](int x, int y) { return (x >> 16) < (y >> 16); });
        unsigned short* out = lv + ebase2[c] + c;
        unsigned short* ends = le + ebase2[c];
        int count = 0, fill = 0;
        for (int o = 0; o < nv; ++o) {
            const int sv = vo[o] & 0xffff;
            const int k1 = vdeg[sv];
            for (int k = sv ? vdeg[sv - 1] : 0; k < k1; ++k) {
                const uint32_t w0 = ve[k];
                if (used[w0 >> 16]) continue;
                used[w0 >> 16] = 1;
                int prev = sv, cur = (int)(w0 & 0xffffu), len = fill;
                uint32_t came = w0 >> 16;
                out[len++] = (unsigned short)sv;
                while (cur != sv) {
                    out[len++] = (unsigned short)cur;
                    uint32_t take = 0xffffffffu;
                    const unsigned long long two = vtwo[cur];
                    if (two != ~0ull) {
                        // the other edge: a walk that reaches it by an unused edge has not been here before
                        take = ((uint32_t)two >> 16) == came ? (uint32_t)(two >> 32) : (uint32_t)two;
                    } else {
                        // an unused edge that does not go straight back, else the first unused one
                        const int q1 = vdeg[cur];
                        for (int q = cur ? vdeg[cur - 1] : 0; q < q1; ++q) {
                            const uint32_t w = ve[q];
                            if (used[w >> 16]) continue;
                            if ((int)(w & 0xffffu) != prev) {
                                take = w;
                                break;
                            }
                            if (take == 0xffffffffu) take = w;
                        }
                        if (take == 0xffffffffu) break;
                    }
                    came = take >> 16;
                    used[came] = 1;
                    prev = cur;
                    cur = (int)(take & 0xffffu);
                }
                if (cur == sv) {
                    fill = len;
                    ends[count++] = (unsigned short)fill;
                }
            }
        }
        nl[c] = count;
    }
    tm.sync();
    const int nloops = team_scan(tm, nl, ncomp);
    each(np, [&](int k) { sh.pr[k].loop0 = nl[sh.pr[k].comp0]; });

    // ---- each loop's sums (src/main.cpp:1027-1040): its terms by lanes, added in loop order by one thread a sum
    int* lrow = reinterpret_cast<int*>(room(4L * nloops));  // first vertex in lv | component: two arrays
    unsigned short* llen = reinterpret_cast<unsigned short*>(room(2L * nloops));
    unsigned short* lcomp = reinterpret_cast<unsigned short*>(room(2L * nloops));
    int* lidx = reinterpret_cast<int*>(room(4L * (nloops + 1)));  // contact flags, then contact numbers
    double* lsum = reinterpret_cast<double*>(room(48L * nloops));
    if (!M.ok) return false;
    each(ncomp, [&](int c) {
        int from = 0;
        for (int k = nl[c]; k < nl[c + 1]; ++k) {
            const int to = le[ebase2[c] + k - nl[c]];
            lrow[k] = ebase2[c] + c + from;
            llen[k] = (unsigned short)(to - from);
            lcomp[k] = (unsigned short)c;
            from = to;
        }
    });
    tm.sync();
    auto edge_terms = [&](const unsigned short* l, int q, int len, double* s6) {
        const double* p0 = V + 3 * l[q];
        const double* p1 = V + 3 * l[q + 1 < len ? q + 1 : 0];
        if constexpr (NPX) {
            for (int k = 0; k < 6; ++k) s6[k] = 0.0;
            np::loop_edge(p0, p1, s6, s6 + 3);
        } else {
            const V3 a0 = team_ld(p0), a1 = team_ld(p1);
            team_st(s6, cross(a0, a1) * 0.5);
            const V3 dx = a1 - a0;
            const double s = dot(a0, a1) + (1.0 / 3.0) * dot(dx, dx);
            team_st(s6 + 3, dx * (-(1.0 / 3.0) * s));
        }
    };
    const int nslot = ne2 + ncomp;  // of lv
    if (L.fits(48L * nslot) || M.fits(48L * nslot)) {
        double* term = reinterpret_cast<double*>(room(48L * nslot));
        for (int k = 0; k < nloops; ++k) {
            const unsigned short* l = lv + lrow[k];
            const int len = llen[k];
            if (len < 3) continue;
            each(len, [&](int q) { edge_terms(l, q, len, term + 6 * (lrow[k] + q)); });
        }
        tm.sync();
        each(6 * nloops, [&](int x) {
            const int k = x / 6, d = x - 6 * k;
            const double* s = term + 6 * lrow[k] + d;
            double r = 0.0;
            if (llen[k] >= 3)
                for (int q = 0; q < llen[k]; ++q) r = r + s[6 * q];
            lsum[x] = r;
        });
    } else {
        each(nloops, [&](int k) {
            double r[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, s[6];
            if (llen[k] >= 3)
                for (int q = 0; q < llen[k]; ++q) {
                    edge_terms(lv + lrow[k], q, llen[k], s);
                    for (int d = 0; d < 6; ++d) r[d] = r[d] + s[d];
                }
            for (int d = 0; d < 6; ++d) lsum[6 * k + d] = r[d];
        });
    }
    tm.sync();
    // ---- which loops are contacts
    auto loop_diag = [&](int k) {
        if (!py) return 0.0;
        const unsigned short* l = lv + lrow[k];
        V3 lo = team_ld(V + 3 * l[0]), hi = lo;
        for (int q = 1; q < llen[k]; ++q) {
            const V3 v = team_ld(V + 3 * l[q]);
            lo = V3{fmin(lo.x, v.x), fmin(lo.y, v.y), fmin(lo.z, v.z)};
            hi = V3{fmax(hi.x, v.x), fmax(hi.y, v.y), fmax(hi.z, v.z)};
        }
        const V3 d = hi - lo;
        if constexpr (NPX) return np::norm3(&d.x);
        return norm(d);
    };
    auto contact_of = [&](int k, double& area, V3& nA, V3& xc0) {
        if (llen[k] < 3) return false;
        const TeamPair& P = sh.pr[cp[lcomp[k]]];
        return team_contact<NPX>(team_ld(lsum + 6 * k), team_ld(lsum + 6 * k + 3), loop_diag(k), py, P.h, P.area_eps,
                                 P.dirAB, area, nA, xc0);
    };
    each(nloops, [&](int k) {
        double area;
        V3 nA, xc0;
        lidx[k] = contact_of(k, area, nA, xc0) ? 1 : 0;
    });
    tm.sync();
    const int nctc = team_scan(tm, lidx, nloops);
    // loop points and tape records: their sizes per loop, then offsets
    const bool tape = a.tape_stage != nullptr;
    int *lpts = nullptr, *ltape = nullptr;
    int npts = 0, ntape = 0;
    if (a.want_pts) {
        lpts = reinterpret_cast<int*>(room(4L * (nloops + 1)));
        if (!M.ok) return false;
        each(nloops, [&](int k) { lpts[k] = lidx[k + 1] > lidx[k] ? llen[k] : 0; });
        tm.sync();
        npts = team_scan(tm, lpts, nloops);
    }
    if (tape) {
        // [L, member offsets (L+1), members as 2*segment + end]
        ltape = reinterpret_cast<int*>(room(4L * (nloops + 1)));
        if (!M.ok) return false;
        each(nloops, [&](int k) {
            int need = 0;
            if (lidx[k + 1] > lidx[k]) {
                const unsigned short* l = lv + lrow[k];
                need = 2 + llen[k];
                for (int q = 0; q < llen[k]; ++q) need += vend[l[q]] - (l[q] ? vend[l[q] - 1] : 0);
            }
            ltape[k] = need;
        });
        tm.sync();
        ntape = team_scan(tm, ltape, nloops);
    }
    // no pair with more points or a longer tape than the warp-per-pair kernel holds
    auto loop_end = [&](int k) { return k + 1 < np ? sh.pr[k + 1].loop0 : nloops; };
    each(np, [&](int k) {
        const int l0 = sh.pr[k].loop0, l1 = loop_end(k), cap2 = 4 * sh.pr[k].n + 64;
        if (a.want_pts && lpts[l1] - lpts[l0] > cap2) sh.bad = 1;
        if (tape && ltape[l1] - ltape[l0] > 2 * (cap2 / 3 + 2) + 2 * cap2 + 8 * sh.pr[k].n + 16) sh.bad = 1;
    });
    tm.sync();
    if (sh.bad) return false;

    // ---- publish
    if (tm.t == 0) {
        sh.cbase = Team::take(a.contact_counter, (unsigned long long)nctc);
        sh.pbase = a.want_pts ? Team::take(a.pts_counter, (unsigned long long)npts) : 0;
        sh.tbase = tape ? Team::take(a.tape_counter, (unsigned long long)ntape) : 0;
    }
    tm.sync();
    const unsigned long long cb = sh.cbase, pb = sh.pbase, tb = sh.tbase;
    const bool cfit = cb + (unsigned long long)nctc <= (unsigned long long)a.contact_cap;
    const bool pfit = pb + (unsigned long long)npts <= (unsigned long long)a.pts_cap;
    const bool tfit = tape && tb + (unsigned long long)ntape <= (unsigned long long)a.tape_cap;
    if (cfit) {
        each(nloops, [&](int k) {
            double area;
            V3 nA, xc0;
            if (lidx[k + 1] == lidx[k]) return;
            contact_of(k, area, nA, xc0);
            const double Fn = 0.5 * a.k * area;
            const V3 FA = py ? nA * Fn : nA * (-Fn);
            const uint64_t o = cb + (unsigned long long)lidx[k];
            double* g = a.cgeom_stage + 20 * o;
            for (int d = 0; d < 6; ++d) g[d] = lsum[6 * k + d];
            team_st(g + 6, xc0);
            team_st(g + 9, nA);
            g[12] = area;
            g[13] = Fn;
            team_st(g + 14, FA);
            team_st(g + 17, FA * -1.0);
            const TeamPair& P = sh.pr[cp[lcomp[k]]];
            int32_t* ci = a.cinfo_stage + 4 * o;
            ci[0] = P.p;
            ci[1] = lidx[k] - lidx[P.loop0];
            ci[2] = llen[k];
            ci[3] = lcomp[k] - P.comp0;
            a.clen_stage[o] = llen[k];
            if (tfit) a.ctape_stage[o] = (int64_t)tb + ltape[k];
        });
    }
    if (a.want_pts && pfit) {
        for (int k = 0; k < nloops; ++k) {
            if (lidx[k + 1] == lidx[k]) continue;
            double* o = a.pts_stage + 3 * (pb + (unsigned long long)lpts[k]);
            each(3 * llen[k], [&](int x) { o[x] = V[3 * lv[lrow[k] + x / 3] + x % 3]; });
        }
    }
    if (tfit) {
        each(nloops, [&](int k) {
            if (lidx[k + 1] == lidx[k]) return;
            const unsigned short* l = lv + lrow[k];
            const int len = llen[k];
            int* r = a.tape_stage + tb + ltape[k];
            const int seg0 = sh.first[cp[lcomp[k]]];
            r[0] = len;
            int mo = 0;
            for (int q = 0; q < len; ++q) {
                r[1 + q] = mo;
                for (int x = l[q] ? vend[l[q] - 1] : 0; x < vend[l[q]]; ++x)
                    r[2 + len + mo++] = 2 * (ord[vmem[x] >> 1] - seg0) + (vmem[x] & 1);
            }
            r[1 + len] = mo;
        });
    }
    if (a.comp_stats) {
        each(ncomp, [&](int c) {
            const TeamPair& P = sh.pr[cp[c]];
            if (c - P.comp0 >= a.comp_stats_cap) return;
            int32_t* cs = a.comp_stats + 3 * ((int64_t)P.p * a.comp_stats_cap + (c - P.comp0));
            cs[0] = comp_off[c + 1] - comp_off[c];
            cs[1] = vbase[c + 1] - vbase[c];
            cs[2] = ebase2[c + 1] - ebase2[c];
        });
    }
    each(np, [&](int k) {
        const TeamPair& P = sh.pr[k];
        const int l0 = P.loop0, l1 = loop_end(k);
        a.pair_stage_off[P.p] = (int64_t)cb + lidx[l0];
        a.pair_pts_stage_off[P.p] = (int64_t)pb + (a.want_pts ? lpts[l0] : 0);
        a.pair_ncontact[P.p] = lidx[l1] - lidx[l0];
        a.pair_npts[P.p] = a.want_pts ? lpts[l1] - lpts[l0] : 0;
        a.pair_ncomp[P.p] = (k + 1 < np ? sh.pr[k + 1].comp0 : ncomp) - P.comp0;
        a.pair_nloop[P.p] = l1 - l0;
    });
    if (tm.t == 0) {
        if (!cfit) Team::flag(a.err, ERR_CONTACT_STAGE);
        if (a.want_pts && !pfit) Team::flag(a.err, ERR_POINT_STAGE);
        if (tape && !tfit) Team::flag(a.err, ERR_TAPE);
    }
    return true;
}

}  // namespace zdx
