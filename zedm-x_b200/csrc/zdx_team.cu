// zdx_team.cu -- the rebuild stage by teams of threads in shared memory (zdx_team.cuh): pairs are sorted into
// classes by their segment count, each class runs a block size and a memory size of its own, a block takes
// packs of pairs, and the pairs no class holds are left to the warp-per-pair kernel of zdx_pair.cu.
//
// What bounds it: latency (chains of shared-memory loads on a warp in the searches and walks, FP64 divides, about
// 40 barriers a pack: 6 of 14 stall cycles an issue), a third of the issue slots used.  The warp-per-pair kernel waited on L1 and L2 for
// the same chains and spent 1,490 warp instructions a segment on scans that this form replaces by lists (about
// 300).  A pack rather than a pair a block: small pairs a warp each had 12 of 32 lanes live and half their stalls
// on instruction fetch, as every warp of an SM was somewhere else in the code.  Three 256-thread blocks an SM
// (80 registers): 128-thread blocks (six an SM, packs of 190 segments) 16.7 ms, two blocks an SM with packs of
// 560 segments 17.0 (256 threads) and 16.9 ms (512) against 16.1 on the pair sweep.
// With the walks, claims and searches of zdx_team.cuh as they are now the first class with 128-thread blocks takes
// 14.4 ms and with 192-thread ones 13.6 against 12.7; the code with its loops rolled up (157 instead of 177 KB) 13.8
// against 13.0.
// Rebuild stage on a B200, warp-per-pair kernel against this: 65,536-pair sweep (103 segments a pair) 27.2 -> 10.1
// ms, 1,500 pairs of 5,120-triangle meshes (400 segments) 6.7 -> 1.6, 16,384 pairs of 320-triangle ones (25)
// 1.79 -> 0.45, 64 mixed pairs 3.85 -> 0.31, one pair of 320-triangle meshes 0.14 -> 0.06.
//
// Compiled with --fmad=false: see zdx_math.cuh.
#include "zdx_team.cuh"

namespace zdx {
namespace {

struct TeamClass {
    int max_seg;   // most segments of a pair of this class
    int pack_seg;  // most segments of a pack
    int bytes;     // shared memory of a block
    int threads;
};
// A pair needs about 150 bytes a segment (205 at most over the pair sweep's mesh sizes; the memories hold 217, 195 and 195
// at the lines, so the top of the larger classes may go to the warp form: none did among pairs of all six modes and
// settings of the tests).  The lines lie where the next larger memory would cost a resident block: three, two and one an
// SM.
__host__ __device__ constexpr TeamClass team_class(int c) {
    return c == 0   ? TeamClass{330, 380, 70 * 1024, 256}
           : c == 1 ? TeamClass{560, 560, 107 * 1024, 256}
                    : TeamClass{1150, 1150, 220 * 1024, 512};
}

__device__ __forceinline__ int64_t items_of(const PairArgs& a) {
    int64_t r = a.item_end - a.item_begin;
    if (a.n_dev && *a.n_dev < r) r = *a.n_dev;
    if (a.order_count && *a.order_count < r) r = *a.order_count;
    return r;
}

// Thread per pair of the order: into its class's list, or (no segment) straight to its result.
__global__ void k_team_classes(PairArgs a, TeamPlan pl) {
    const int lane = threadIdx.x & 31;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int cls = -1, p = 0;
    if (i < items_of(a)) {
        p = a.order[a.item_begin + i];
        const int n = a.pair_nseg[p];
        if (a.pair_status[p] != 0) {
            cls = TEAM_CLASSES;
        } else if (n == 0) {
            a.pair_stage_off[p] = 0;
            a.pair_pts_stage_off[p] = 0;
            a.pair_ncontact[p] = 0;
            a.pair_npts[p] = 0;
            a.pair_ncomp[p] = 0;
            a.pair_nloop[p] = 0;
        } else {
            cls = 0;
            while (cls < TEAM_CLASSES && n > team_class(cls).max_seg) ++cls;
        }
    }
    for (int c = 0; c <= TEAM_CLASSES; ++c) {
        const unsigned b = __ballot_sync(0xffffffffu, cls == c);
        if (!b) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(pl.counts + c, __popc(b));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (cls == c) pl.lists[c * pl.stride + base + __popc(b & ((1u << lane) - 1u))] = p;
    }
}

// A block claims items of its class's list a few at a time and packs as many of them as its memory takes.  A
// pack that is not held is taken again pair by pair; a pair that is not held goes to the last list.
template <int T, int BLOCKS, bool NPX>
__global__ void __launch_bounds__(T, BLOCKS) k_rebuild_team(PairArgs a, TeamPlan pl, int cls, int pack_seg, int bytes) {
    extern __shared__ __align__(16) char team_mem[];
    __shared__ TeamShared sh;
    DevTeam<T> tm;
    tm.t = threadIdx.x;
    tm.sh = &sh;
    const int count = pl.counts[cls];
    // A claim is a number of items that are `claims` apart in the list (which is sorted by cost, so that claims are
    // alike): one claim a block where that is a few items (a pack takes the time of its longest chains, whether
    // it holds one small pair or eight), two or more a block otherwise.
    const int blocks = (int)gridDim.x, per = (count + blocks - 1) / blocks;
    const int claim = max(1, min(TEAM_PACK, per <= 4 ? per : (per + 1) / 2));
    const int claims = (count + claim - 1) / claim;
    const int32_t* list = pl.lists + cls * pl.stride;
    if (threadIdx.x == 0) sh.from = sh.to = 0;
    int again = 0, held = 0;  // pairs of a refused pack still to be taken alone
    for (;;) {
        tm.sync();
        if (again < held) {
            if (threadIdx.x == 0) {
                sh.pr[0].p = sh.claimed[again];
                sh.np = 1;
            }
            ++again;
        } else if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int from = sh.from, to = sh.to;
            if (from >= to) {  // items from, from + claims, ... below to
                if (lane == 0) from = atomicAdd(pl.counts + 8 + cls, 1);
                from = __shfl_sync(0xffffffffu, from, 0);
                to = from < claims ? count : from;
            }
            const int64_t at = from + (int64_t)lane * claims;
            const bool live = at < to;
            const int p = live ? list[at] : 0;
            int sum = live ? a.pair_nseg[p] : 0;
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += y;
            }
            // the first always fits; a bit for each of the lanes that do with all before them
            const int np = __popc(__ballot_sync(0xffffffffu, live && (lane == 0 || sum <= pack_seg)));
            if (lane < np) sh.pr[lane].p = sh.claimed[lane] = p;
            if (lane == 0) {
                sh.np = np;
                sh.from = from + np * claims;
                sh.to = to;
            }
        }
        tm.sync();
        const int np = sh.np;
        if (np == 0) break;
        if (team_rebuild<DevTeam<T>, NPX>(tm, a, np, team_mem, bytes)) continue;
        if (np > 1) {
            again = 0;
            held = np;
        } else if (threadIdx.x == 0) {
            pl.lists[TEAM_CLASSES * pl.stride + atomicAdd(pl.counts + TEAM_CLASSES, 1)] = sh.pr[0].p;
        }
    }
}

template <int C, int BLOCKS, bool NPX>
void launch_class(const PairArgs& a, const TeamPlan& pl, int sms, int64_t most, cudaStream_t s) {
    constexpr TeamClass c = team_class(C);
    auto k = k_rebuild_team<c.threads, BLOCKS, NPX>;
    // per device and cheap: set on every launch
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, c.bytes);
    cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    const int64_t grid = (int64_t)sms * BLOCKS;
    k<<<(unsigned)(most < grid ? most : grid), c.threads, c.bytes, s>>>(a, pl, C, c.pack_seg, c.bytes);
}

// The classes share nothing but counters, and each ends with the chains of its last pairs on an idle chip: with a
// second stream the classes of large pairs run beside the first.  Rebuild stage with one stream and with two: 65,536-pair
// sweep 11.1 and 10.1 ms, 1,500 pairs of 5,120-triangle meshes 1.82 and 1.59, 64 mixed pairs 0.49 and 0.31.  A call
// of one class keeps to one stream (a second one in the context cost the single-pair call 0.06 of 0.45 ms).
template <bool NPX>
int launch_classes(const PairArgs& a, const TeamPlan& pl, int sms, int64_t most, int nmax, cudaStream_t s,
                   const TeamSide* side) {
    // blocks an SM holds: 227 KB over the class's memory, 5 KB of its own and the system's
    const int n = team_classes_of(nmax);
    const cudaStream_t s2 = side ? side->stream : s;
    if (side) {
        cudaEventRecord(side->ev[0], s);
        cudaStreamWaitEvent(s2, side->ev[0], 0);
    }
    if (n > 2) launch_class<2, 1, NPX>(a, pl, sms, most, s2);
    if (n > 1) launch_class<1, 2, NPX>(a, pl, sms, most, s2);
    if (n > 0) launch_class<0, 3, NPX>(a, pl, sms, most, s);  // none: no pair has a segment
    if (side) {
        cudaEventRecord(side->ev[1], s2);
        cudaStreamWaitEvent(s, side->ev[1], 0);
    }
    return n;
}

}  // namespace

int team_classes_of(int nmax) { return nmax <= 0 ? 0 : nmax <= team_class(0).max_seg ? 1 : nmax <= team_class(1).max_seg ? 2 : 3; }

int launch_rebuild_teams(const PairArgs& a, const TeamPlan& pl, int sms, int64_t most, int nmax, cudaStream_t s,
                         const TeamSide* side) {
    if (most <= 0) return 0;
    k_team_classes<<<(unsigned)((most + 255) / 256), 256, 0, s>>>(a, pl);
    return 1 + (a.mode == 2 ? launch_classes<true>(a, pl, sms, most, nmax, s, side)
                            : launch_classes<false>(a, pl, sms, most, nmax, s, side));
}

cudaError_t load_rebuild_teams() {
    cudaFuncAttributes f;
    const void* ks[4] = {(const void*)k_team_classes, (const void*)k_rebuild_team<team_class(0).threads, 3, false>,
                         (const void*)k_rebuild_team<team_class(1).threads, 2, false>,
                         (const void*)k_rebuild_team<team_class(2).threads, 1, false>};
    for (const void* k : ks)
        if (cudaError_t e = cudaFuncGetAttributes(&f, k)) return e;
    return cudaSuccess;
}

}  // namespace zdx
