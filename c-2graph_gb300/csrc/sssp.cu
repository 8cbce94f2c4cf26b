// Single-query SSSP for sm_103a: one persistent cooperative launch per query.
//
// Replaces CalcuSSSP (reference src/sssp/base/Main.cu:109-356 and
// src/sssp/purn/Main.cu:136-393).  Same result: the int32 shortest-distance fixed point
// of dis[source] = 0 plus the pruned-record seeds (sssp-purn), unreachable = 1999999999.
// Different schedule:
//   * frontier = sparse list of (vertex, edge base) appended by warp-aggregated atomics
//     when a distance improves (no O(V) isactive sweep, src/sssp/purn/Main.cu:350-377);
//   * expansion is edge-tiled: the frontier's out-edges form one index range [0, T),
//     each warp takes tiles of 2^log_tile edges from a dynamic counter, so low-degree
//     vertices share a tile (thread-per-edge), high-degree vertices span many tiles
//     (many warps per vertex), and every lane reads consecutive (target, weight) pairs;
//   * relaxation is an L2 read guarding int32 atomicMin (src/sssp/purn/Main.cu:257-260);
//   * optional near/far split (delta-stepping): improvements at or above the bucket
//     threshold go to a far pile that is filtered into the frontier when the near
//     frontier runs dry;
//   * one bounded grid barrier per round instead of four unbounded spins.
#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>

#include "device_common.cuh"
#include "internal.h"

namespace c2g {

struct SsspParams {
    const int* row;
    const int2* adj;
    unsigned E;
    int V;
    int* dist;
    int* stamp;
    int* farstamp;
    int stamp_extent;  // entries of stamp/farstamp cleared when the round tags restart (>= V)
    int2* q[2];
    int* mark[2];
    int* far[3];
    TraversalCtl* ctl;
    StampState* st;
    int source;
    const int* seed_v;
    const int* seed_w;
    int n_seeds;
    int delta;
    int log_tile;
    int max_iter;
    unsigned mark_cap;
    unsigned long long barrier_ns;
    unsigned bar_extra;  // > 0: barriers wait for blocks that do not exist (watchdog test)
};

__device__ __forceinline__ FrontierOut sssp_out(const SsspParams& p, int buf, int slot) {
    FrontierOut o;
    o.q = p.q[buf];
    o.val = nullptr;
    o.mark = p.mark[buf];
    o.ctr = &p.ctl->qctr[slot];
    o.cap = (unsigned)p.V;
    o.mark_cap = p.mark_cap;
    o.log_tile = p.log_tile;
    o.flags = &p.ctl->flags;
    return o;
}

// Near-frontier candidate: dedup by round tag, drop vertices without out-edges.
__device__ __forceinline__ bool claim_near(const SsspParams& p, int c, int tag, int& deg) {
    if (ldcg(p.stamp + c) == tag || atomicExch(p.stamp + c, tag) == tag) return false;
    deg = __ldg(p.row + c + 1) - __ldg(p.row + c);
    return deg > 0;
}

// Far pile stage of one warp: staged ids plus the minimum distance staged so far.
struct FarStage {
    WarpStage st;
    int fmin;
};

// Warp-collective: stage lanes with `want` for far pile fb (deduplicated per epoch when
// `dedup`), tracking the minimum pushed distance.
__device__ __forceinline__ void far_stage(const SsspParams& p, FarStage& fs, int fb, bool want, int c, int d,
                                          int epoch, bool dedup) {
    if (want && dedup) {
        if (ldcg(p.farstamp + c) == epoch || atomicExch(p.farstamp + c, epoch) == epoch) want = false;
    }
    if (__ballot_sync(kFull, want) == 0) return;
    int mn = want ? d : INT_MAX;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, o));
    fs.fmin = min(fs.fmin, mn);
    list_stage_push(fs.st, p.far[fb], &p.ctl->farctr[fb], (unsigned)p.V, &p.ctl->flags, want, c);
}

__device__ __forceinline__ void far_flush(const SsspParams& p, FarStage& fs, int fb) {
    list_stage_flush(fs.st, p.far[fb], &p.ctl->farctr[fb], (unsigned)p.V, &p.ctl->flags);
    if ((threadIdx.x & 31) == 0 && fs.fmin != INT_MAX) atomicMin(&p.ctl->farmin[fb], fs.fmin);
    fs.fmin = INT_MAX;
}

constexpr int kSsspUnroll = 4;  // edges in flight per lane

template <bool kDelta>
__device__ __forceinline__ void sssp_expand(const SsspParams& p, int buf, unsigned F, unsigned T, int tag_next,
                                            int thresh, int fb, int epoch, const FrontierOut& nout,
                                            WarpStage& fst, FarStage& far) {
    constexpr int U = kSsspUnroll;
    walk_frontier_edges<U>(
        p.q[buf], p.mark[buf], p.row, F, T, p.log_tile, p.mark_cap, (unsigned)p.V, p.E, &p.ctl->flags,
        [&](int v, unsigned) { return ldcg(p.dist + v); },  // snapshot distance of the owner
        [&](const bool* ok, const unsigned* idx, const int* du) {
            int c[U], nd[U], cur[U];
            // U independent edge loads, then U independent distance reads.
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int2 ew = ok[u] ? __ldg(p.adj + idx[u]) : make_int2(0, 0);
                c[u] = ew.x;
                nd[u] = du[u] + ew.y;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) cur[u] = ok[u] ? ldcg(p.dist + c[u]) : INT_MIN;
            bool near[U], farp[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                near[u] = farp[u] = false;
                if (nd[u] < cur[u]) {  // an L2 read guards the atomic
                    const int old = atomicMin(p.dist + c[u], nd[u]);
                    if (nd[u] < old) {
                        if (!kDelta || nd[u] < thresh)
                            near[u] = true;
                        else
                            farp[u] = true;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                int deg = 0;
                const bool want = near[u] && claim_near(p, c[u], tag_next, deg);
                stage_push(fst, nout, want, c[u], deg, 0.f);
                if (kDelta) far_stage(p, far, fb, farp[u], c[u], nd[u], epoch, true);
            }
        });
    stage_flush(fst, nout);
    if (kDelta) far_flush(p, far, fb);
}

template <bool kDelta>
__global__ void __launch_bounds__(512, 2) sssp_persistent(const SsspParams p) {
    TraversalCtl* ctl = p.ctl;
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(&ctl->bar_count);
    grid_sync_init();
    int* flags = &ctl->flags;
    const int lane = threadIdx.x & 31;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nthreads = gridDim.x * blockDim.x;
    const unsigned gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const unsigned V = (unsigned)p.V;
    __shared__ StageSmem sm;
    const int wib = threadIdx.x >> 5;
    WarpStage fst{sm.v0[wib], sm.d0[wib], nullptr, 0};
    FarStage far{WarpStage{sm.v1[wib], nullptr, nullptr, 0}, INT_MAX};
    unsigned long long tph = globaltimer_ns();

    int sbase = p.st->stamp_base;
    int ebase = p.st->epoch_base;
    const bool reset = sbase > (1 << 29) || ebase > (1 << 29);
    if (reset) sbase = ebase = 0;

    // Init: dis = INF (src/sssp/purn/Main.cu:144-156).
    for (unsigned v = gtid; v < V; v += nthreads) p.dist[v] = kInfDist;
    // Restarting tags clear every stamp the array holds, not only this graph's V: an
    // array shared by calls on graphs of different sizes keeps older tags beyond V,
    // which a later, larger graph would read as current.
    if (reset)
        for (unsigned v = gtid; v < (unsigned)p.stamp_extent; v += nthreads) {
            p.stamp[v] = -1;
            p.farstamp[v] = -1;
        }
    if (gtid == 0) ctl->farmin[0] = ctl->farmin[1] = ctl->farmin[2] = INT_MAX;
    if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;

    // Source and pruned-record seeds (src/sssp/purn/Main.cu:160-181).
    if (gtid == 0) {
        atomicMin(p.dist + p.source, 0);
        ctl->seeds = p.n_seeds;
    }
    for (unsigned i = gtid; i < (unsigned)p.n_seeds; i += nthreads) atomicMin(p.dist + p.seed_v[i], p.seed_w[i]);
    if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;

    // Round-1 frontier: the seeds and the source, deduplicated.
    {
        const int tag = sbase + 1;
        const FrontierOut out = sssp_out(p, 1, 1);
        const unsigned n = (unsigned)p.n_seeds + 1;
        for (unsigned b = gwarp * 32; b < n; b += nwarps * 32) {
            const unsigned i = b + (unsigned)lane;
            bool want = false;
            int v = 0, deg = 0;
            if (i < n) {
                v = (i < (unsigned)p.n_seeds) ? p.seed_v[i] : p.source;
                want = claim_near(p, v, tag, deg);
            }
            stage_push(fst, out, want, v, deg, 0.f);
        }
        stage_flush(fst, out);
    }
    if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
    phase_mark(ctl->phase_ns, tph, 0);

    int cur = 1, fb = 0, epoch = ebase + 1, iters = 0;
    int thresh = kDelta ? p.delta : INT_MAX;
    for (;;) {
        const unsigned long long c = ldcg(&ctl->qctr[cur % 3]);
        const unsigned F = (unsigned)(c >> 32), T = (unsigned)c;
        if (F == 0) {
            if (!kDelta) break;
            const unsigned fc = ldcg(&ctl->farctr[fb]);
            if (fc == 0) break;
            // Next bucket: at least thresh + delta, and past the far pile's minimum.
            const int fm = ldcg(&ctl->farmin[fb]);
            long long nt = (long long)thresh + p.delta;
            const long long jump = ((long long)fm / p.delta + 1) * (long long)p.delta;
            if (jump > nt) nt = jump;
            if (nt > INT_MAX) nt = INT_MAX;
            const int fdst = (fb + 1) % 3;
            if (gtid == 0) {
                const int fold = (fb + 2) % 3;  // read by the previous filter, free now
                ctl->farctr[fold] = 0;
                ctl->farmin[fold] = INT_MAX;
                ctl->qctr[(cur + 2) % 3] = 0ull;
                ctl->tilectr[(cur + 2) % 3] = 0u;
            }
            // The filter's frontier is the next round's (slot cur + 1): every thread has
            // read slot cur above to see it empty, and a late reader must not see these
            // appends there (it would take the expansion branch and skip its share of
            // the pile).
            const FrontierOut out = sssp_out(p, (cur + 1) & 1, (cur + 1) % 3);
            const int tag = sbase + cur + 1;
            for (unsigned b = gwarp * 32; b < fc; b += nwarps * 32) {
                const unsigned i = b + (unsigned)lane;
                bool near = false, keep = false;
                int v = 0, deg = 0, d = 0;
                if (i < fc) {
                    v = ldcg(p.far[fb] + i);
                    d = ldcg(p.dist + v);
                    if (d >= thresh) {
                        if (d < (int)nt)
                            near = claim_near(p, v, tag, deg);
                        else {
                            keep = true;
                            p.farstamp[v] = epoch + 1;
                        }
                    }
                }
                stage_push(fst, out, near, v, deg, 0.f);
                far_stage(p, far, fdst, keep, v, d, epoch + 1, false);
            }
            stage_flush(fst, out);
            far_flush(p, far, fdst);
            thresh = (int)nt;
            fb = fdst;
            ++epoch;
            if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
            phase_mark(ctl->phase_ns, tph, 1);
            ++cur;
            continue;
        }
        if (++iters > p.max_iter) {
            if (gtid == 0) atomicOr(flags, C2G_FLAG_ITER_CAP);
            break;
        }
        if (gtid == 0) {
            ctl->qctr[(cur + 2) % 3] = 0ull;
            ctl->tilectr[(cur + 2) % 3] = 0u;
            ctl->popped += F;
            ctl->relaxed += T;
        }
        const FrontierOut nout = sssp_out(p, (cur + 1) & 1, (cur + 1) % 3);
        sssp_expand<kDelta>(p, cur & 1, F, T, sbase + cur + 1, thresh, fb, epoch, nout, fst, far);
        if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
        phase_mark(ctl->phase_ns, tph, 2);
        ++cur;
    }
    if (gtid == 0) {
        ctl->iterations = iters;
        p.st->stamp_base = sbase + cur + 2;
        p.st->epoch_base = epoch + 2;
    }
}

// Bellman-Ford rounds (delta = 0), each a push or a pull.
//
// Push: the frontier is a list; a relaxation that improves a distance issues red.min on it and
// red.or of the vertex's bit into a V-bit map; neither waits for a return value, so the
// relaxation path has no atomic round trip (the list kernel above needs the atomicMin result
// and a round-tag exchange per improved vertex).  A sweep over the V/32 map words builds
// the next frontier in vertex order (entries, edge-base prefix, tile markers) and clears the
// words: two grid barriers per round.
//
// Pull: every vertex v reads its in-edges, ordered by weight (in_edges.cu), as long as
// w + (smallest frontier distance) < dist[v]: no later edge can improve v.  A push of a dense
// frontier is bound by one random L2 read per out-edge of the frontier; in a pull most rows
// end after one or two groups of 4 edges, hub rows too (their distance is small).  The warp
// that pulls v is the only writer of dist[v] in the round, so it stores without atomics,
// writes the map word of its 32 vertices and counts the next frontier: a pull needs no list,
// and one barrier.
//
// Any order of relaxations reaches the same fixed point, so the rounds mix freely.
constexpr int kSweepGroup = 4;  // map words whose row bounds are loaded together
constexpr int kBitsThreads = 512;  // block size of the bitmap kernel (its own launch geometry)
constexpr int kBitsBlocksPerSm = 2;
// Round-robin tiles in the expansion: a dynamic tile queue measured slower here (2.74 vs
// 2.20 ms per scale-22 query).
constexpr bool kBitsDynTiles = false;
// Swept at scale 22 / 16 (1.05 ms, 133 us): 1, 2 or 3 words at a time, 2 or 4 lane groups, 1.05 - 1.13 ms.
constexpr int kPullWords = 2;    // map words a warp pulls at a time
constexpr int kLaneGroups = 2;   // groups of 4 in-edges a lane reads before the warp shares the rest
constexpr int kWarpGroups = 16;  // rows that need more groups than this go to the whole grid
constexpr int kPullTile = 6;     // log2 of the groups per warp tile of those rows

// In-edge rows and round rule of the kernel.
struct SsspPull {
    const int* row;   // in-edge rows, or nullptr: push only
    const int2* adj;
    int shift;           // weights are ordered up to their low `shift` bits
    unsigned pull_min;   // a round pulls when its frontier has more out-edges (~0: never)
    int always;          // every round pulls: no map, no list
    unsigned* bits[2];   // maps of the frontiers of the rounds of each parity
    double* long_at;     // long rows: (distance to count from << 32) | first group, beside their queue entry
    int* long_mark;      // tile owners over their groups
    unsigned long_tiles;
};

// Warp-collective: the frontier list of a round from its map; the words are cleared.
__device__ __forceinline__ void bits_sweep(const SsspParams& p, unsigned* bits, const FrontierOut& out,
                                           WarpStage& fst, unsigned gwarp, unsigned nwarps, int lane) {
    const unsigned V = (unsigned)p.V;
    const unsigned nw = (V + 31u) >> 5;
    for (unsigned b = gwarp * 32u; b < nw; b += nwarps * 32u) {
        const unsigned wi = b + (unsigned)lane;
        const unsigned m = wi < nw ? ldcg(bits + wi) : 0u;
        if (m) bits[wi] = 0u;
        unsigned nz = __ballot_sync(kFull, m != 0u);
        while (nz) {
            int ks[kSweepGroup], deg[kSweepGroup];
            bool set[kSweepGroup];
#pragma unroll
            for (int u = 0; u < kSweepGroup; ++u) {
                ks[u] = nz ? __ffs(nz) - 1 : -1;
                nz &= nz - 1u;
            }
#pragma unroll
            for (int u = 0; u < kSweepGroup; ++u) {
                const unsigned mk = ks[u] < 0 ? 0u : (unsigned)__shfl_sync(kFull, (int)m, ks[u] < 0 ? 0 : ks[u]);
                const unsigned v = ((b + (unsigned)(ks[u] < 0 ? 0 : ks[u])) << 5) + (unsigned)lane;
                set[u] = (mk >> lane) & 1u;
                deg[u] = set[u] ? __ldg(p.row + v + 1) - __ldg(p.row + v) : 0;
            }
#pragma unroll
            for (int u = 0; u < kSweepGroup; ++u) {
                if (ks[u] < 0) break;  // warp-uniform
                const unsigned v = ((b + (unsigned)ks[u]) << 5) + (unsigned)lane;
                stage_push(fst, out, set[u] && deg[u] > 0, (int)v, deg[u], 0.f);
            }
        }
    }
    stage_flush(fst, out);
}

// A block's part of a round's totals, added to the round's counters once per block.
struct RoundShare {
    unsigned long long count;  // (vertices with out-edges << 32) | out-edges, of the improved vertices
    int fmin;                  // smallest improved distance
};

// Add a warp's totals of a round to its block's, and the block's to the round's counters
// (every warp of the grid adding to one address took longer than a short round).
__device__ __forceinline__ void round_totals(TraversalCtl* ctl, int slot, RoundShare* share,
                                             unsigned long long count, int fnew, int lane) {
    for (int o = 16; o >= 1; o >>= 1) count += __shfl_xor_sync(kFull, count, o);
    fnew = __reduce_min_sync(kFull, fnew);
    if (lane == 0) {
        if (count) atomicAdd(&share->count, count);
        if (fnew != INT_MAX) atomicMin(&share->fmin, fnew);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (share->count) atomicAdd(&ctl->pcount[slot], share->count);
        if (share->fmin != INT_MAX) atomicMin(&ctl->farmin[slot], share->fmin);
        *share = RoundShare{0ull, INT_MAX};
    }
}

// A group of 4 in-edges (source, weight): the smallest candidate distance below b among the
// edges that can improve it (weight below lim).
__device__ __forceinline__ int pull_edges(const int* dist, const int4& x, const int4& y, int lim, int b) {
    // Read through L1: other warps lower distances during the round, and either value is a
    // valid upper bound (a lowered source is in the next frontier); the barrier's acquire
    // makes the next round read anew.
    const int d0 = x.y < lim ? __ldca(dist + x.x) : kInfDist;
    const int d1 = x.w < lim ? __ldca(dist + x.z) : kInfDist;
    const int d2 = y.y < lim ? __ldca(dist + y.x) : kInfDist;
    const int d3 = y.w < lim ? __ldca(dist + y.z) : kInfDist;
    // an edge that cannot improve has weight up to INT_MAX (the padding): no sum of its own
    if (x.y < lim) b = min(b, d0 + x.y);
    if (x.w < lim) b = min(b, d1 + x.w);
    if (y.y < lim) b = min(b, d2 + y.y);
    if (y.w < lim) b = min(b, d3 + y.w);
    return b;
}

__device__ __forceinline__ int pull_group(const SsspPull& in, const int* dist, int i, int lim, int b, int* last) {
    const int4 x = __ldg(reinterpret_cast<const int4*>(in.adj + i));
    const int4 y = __ldg(reinterpret_cast<const int4*>(in.adj + i + 2));
    *last = (y.w >> in.shift) << in.shift;
    return pull_edges(dist, x, y, lim, b);
}

// Queue of a pull round's long rows: (vertex, exclusive prefix of the groups to read), with the first group in
// long_at beside the distance that the second part may count the vertex from (-1: the first part lowered the
// distance and has counted it).  It uses the list buffers, idle in a pull round.
__device__ __forceinline__ FrontierOut pull_long_out(const SsspParams& p, const SsspPull& in, int parity) {
    FrontierOut o;
    o.q = p.q[0];
    o.val = nullptr;
    o.vald = in.long_at;
    o.mark = in.long_mark;
    o.ctr = &p.ctl->lctr[parity];
    o.cap = (unsigned)p.V;
    o.mark_cap = in.long_tiles;
    o.log_tile = kPullTile;
    o.flags = &p.ctl->flags;
    return o;
}

// What is left of a word's rows after their first group (b0: the distances before it): lanes read on up to kLaneGroups
// groups; a row that needs more finds by bisection how many groups can still improve it.  Up to
// kWarpGroups the warp reads together, all rows' groups in one sequence; longer rows are
// queued for the whole grid.
__device__ __forceinline__ int pull_rest(const SsspParams& p, const SsspPull& in, int fmin, unsigned v, int b0, int b,
                                      int i, int e, bool more, int* best, WarpStage& lst, const FrontierOut& lout, int lane) {
    int last = INT_MIN;
#pragma unroll 1
    for (int s = 1; s < kLaneGroups; ++s) {
        if (more) {
            b = pull_group(in, p.dist, i, b - fmin, b, &last);
            i += 4;
        }
        more = more && i < e && last < b - fmin;
        if (!__any_sync(kFull, more)) return b;
    }
    // groups [0, n) from i on start below the limit (their first weight, rounded down)
    int n = 0;
    if (more) {
        int hi = (e - i) >> 2;
        while (n < hi) {  // the first group at or above the limit is in [n, hi]: three probes at a time
            const int q = (hi - n) >> 2, m1 = n + q, m2 = m1 + q, m3 = m2 + q;
            const bool b1 = ((__ldg(in.adj + i + 4 * m1).y >> in.shift) << in.shift) < b - fmin;
            const bool b2 = ((__ldg(in.adj + i + 4 * m2).y >> in.shift) << in.shift) < b - fmin;
            const bool b3 = ((__ldg(in.adj + i + 4 * m3).y >> in.shift) << in.shift) < b - fmin;
            if (!b1) hi = m1;
            else if (!b2) { n = m1 + 1; hi = m2; }
            else if (!b3) { n = m2 + 1; hi = m3; }
            else n = m3 + 1;
        }
    }
    const bool queued = n > kWarpGroups;
    const unsigned from = b < b0 ? ~0u : (unsigned)b;
    stage_push(lst, lout, queued, (int)v, n, 0.f,
               __longlong_as_double((long long)(((unsigned long long)from << 32) | (unsigned)i)));
    if (queued) n = 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    const unsigned base = (unsigned)(incl - n), total = (unsigned)__shfl_sync(kFull, incl, 31);
    best[lane] = b;
    __syncwarp();
    for (unsigned g = (unsigned)lane; g - (unsigned)lane < total; g += 32u) {
        const int k = owner_lane(base, g);
        const int ki = __shfl_sync(kFull, i, k);
        const unsigned kb = (unsigned)__shfl_sync(kFull, (int)base, k);
        if (g < total) {
            const int bk = *(volatile int*)(best + k);
            int unused;
            const int nb = pull_group(in, p.dist, ki + 4 * (int)(g - kb), bk - fmin, bk, &unused);
            if (nb < bk) atomicMin(best + k, nb);
        }
    }
    __syncwarp();
    b = best[lane];
    __syncwarp();
    return b;
}

// First part of a pull round.  Each warp takes map words (32 vertices, one per lane),
// kPullWords at a time so that their first groups' loads are in flight together: at scale 22
// a pull reads about one group and one source distance per vertex, so it is bound by the chain
// word -> group -> sources, not by bytes.  Consecutive words go to different blocks and the
// stride over words is odd: the busiest vertices of a skewed graph have neighbouring ids and
// ids that are multiples of powers of two (with an even stride 170 of 4,864 warps took
// 113 us where the average was 42 us).  The rows that need more groups follow in pull_rest.
__device__ __forceinline__ void sssp_pull(const SsspParams& p, const SsspPull& in, int fmin, unsigned* bits_cur,
                                          unsigned* bits_next, int* best, WarpStage& lst, const FrontierOut& lout,
                                          unsigned long long& count, int& fnew, int lane, int wib) {
    const unsigned V = (unsigned)p.V;
    const unsigned nw = (V + 31u) >> 5;
    const unsigned nwarps = (((gridDim.x * blockDim.x) >> 5) - 1u) | 1u;  // odd
    const unsigned wfirst = (unsigned)wib * gridDim.x + blockIdx.x;
    for (unsigned w0 = wfirst < nwarps ? wfirst : nw; w0 < nw; w0 += kPullWords * nwarps) {
        int b0[kPullWords], b[kPullWords], i[kPullWords], e[kPullWords], last[kPullWords], deg[kPullWords];
        // first groups of all words, their loads in flight together
#pragma unroll
        for (int u = 0; u < kPullWords; ++u) {
            const unsigned v = ((w0 + u * nwarps) << 5) + (unsigned)lane;
            const bool in_range = w0 + u * nwarps < nw && v < V;
            b0[u] = in_range ? ldcg(p.dist + v) : INT_MIN;
            i[u] = in_range ? __ldg(in.row + v) : 0;
            e[u] = in_range ? __ldg(in.row + v + 1) : 0;
        }
        int4 x[kPullWords], y[kPullWords];
#pragma unroll
        for (int u = 0; u < kPullWords; ++u) {
            const bool go = i[u] < e[u] && b0[u] > fmin;
            x[u] = go ? __ldg(reinterpret_cast<const int4*>(in.adj + i[u])) : make_int4(0, INT_MAX, 0, INT_MAX);
            y[u] = go ? __ldg(reinterpret_cast<const int4*>(in.adj + i[u] + 2)) : make_int4(0, INT_MAX, 0, INT_MAX);
            if (!go) e[u] = i[u];
        }
#pragma unroll
        for (int u = 0; u < kPullWords; ++u) {
            b[u] = pull_edges(p.dist, x[u], y[u], b0[u] - fmin, b0[u]);
            last[u] = (y[u].w >> in.shift) << in.shift;
            i[u] += 4;
        }
#pragma unroll
        for (int u = 0; u < kPullWords; ++u) {
            const bool more = i[u] < e[u] && last[u] < b[u] - fmin;
            if (__any_sync(kFull, more))
                b[u] = pull_rest(p, in, fmin, ((w0 + u * nwarps) << 5) + (unsigned)lane, b0[u], b[u], i[u], e[u], more,
                                 best, lst, lout, lane);
        }
#pragma unroll
        for (int u = 0; u < kPullWords; ++u) {
            const unsigned v = ((w0 + u * nwarps) << 5) + (unsigned)lane;
            deg[u] = 0;
            if (b[u] < b0[u]) {
                p.dist[v] = b[u];
                deg[u] = __ldg(p.row + v + 1) - __ldg(p.row + v);
                fnew = min(fnew, b[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kPullWords; ++u) {
            if (deg[u] > 0) count += (1ull << 32) | (unsigned)deg[u];
            if (!in.always && w0 + u * nwarps < nw) {
                const unsigned m = __ballot_sync(kFull, deg[u] > 0);
                if (lane == 0) {
                    bits_next[w0 + u * nwarps] = m;
                    bits_cur[w0 + u * nwarps] = 0u;  // this round's frontier, if it was not listed
                }
            }
        }
    }
    stage_flush(lst, lout);
}

// What a warp keeps of its word for all rounds (sssp_pull_kept).
struct KeptWord {
    int4 x[32], y[32];  // the rows' first groups
    int2 rest[32];      // first in-edge behind them, end
    int deg[32];        // out-degrees
};

__device__ __forceinline__ void kept_load(const SsspParams& p, const SsspPull& in, KeptWord& k, int lane, int wib) {
    const unsigned v = (((unsigned)wib * gridDim.x + blockIdx.x) << 5) + (unsigned)lane;
    int i = 0, e = 0, deg = 0;
    int4 x = make_int4(0, INT_MAX, 0, INT_MAX), y = x;
    if (v < (unsigned)p.V) {
        i = __ldg(in.row + v);
        e = __ldg(in.row + v + 1);
        deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
        if (i < e) {
            x = __ldg(reinterpret_cast<const int4*>(in.adj + i));
            y = __ldg(reinterpret_cast<const int4*>(in.adj + i + 2));
        }
    }
    k.x[lane] = x;
    k.y[lane] = y;
    k.rest[lane] = make_int2(i + 4, e);
    k.deg[lane] = deg;
}

// The first part on a graph with at most one word per warp.  Its rounds are chains of loads (counts, distances
// and row bounds, first groups, sources, out-degrees) between barriers, so the word's first groups and
// degrees stay in shared memory, and its distances, which only this warp and the second part write, in b (read
// anew where stale: rows that may have been queued).  A query at scale 12 (8 edges per vertex) 89.6 -> 74.6 us,
// scale 16 pruned 133 -> 122, 100,003 uniform vertices 207 -> 178; what is left of a round's 6 us is the
// barrier, the counts, one gather and the rows that need more than a group.
__device__ __forceinline__ void sssp_pull_kept(const SsspParams& p, const SsspPull& in, int fmin, const KeptWord& k,
                                               int& b, bool& stale, int* best, WarpStage& lst,
                                               const FrontierOut& lout, unsigned long long& count, int& fnew,
                                               int lane, int wib) {
    const unsigned w = (unsigned)wib * gridDim.x + blockIdx.x;
    const unsigned v = (w << 5) + (unsigned)lane;
    if ((w << 5) < (unsigned)p.V) {
        if (stale) b = v < (unsigned)p.V ? ldcg(p.dist + v) : INT_MIN;
        const int b0 = b;
        const int4 x = k.x[lane], y = k.y[lane];
        const int2 rest = k.rest[lane];
        // (a row that is done, or empty, has nothing below the limit)
        const bool go = b0 > fmin;
        if (go) b = pull_edges(p.dist, x, y, b0 - fmin, b0);
        const int last = (y.w >> in.shift) << in.shift;
        const bool more = go && rest.x < rest.y && last < b - fmin;
        stale = more && rest.y - rest.x > 4 * kWarpGroups;
        if (__any_sync(kFull, more)) b = pull_rest(p, in, fmin, v, b0, b, rest.x, rest.y, more, best, lst, lout, lane);
        if (b < b0) {
            p.dist[v] = b;
            fnew = min(fnew, b);
            const int deg = k.deg[lane];
            if (deg > 0) count += (1ull << 32) | (unsigned)deg;
        }
    }
    stage_flush(lst, lout);
}

// Second part, after a barrier, when rows were queued (a hub row that nothing has reached yet needs
// all its 100,000 edges: read by its warp alone that took 1.07 ms of a scale-22 query): warps
// take tiles of their groups, and a row's parts meet in atomicMin.  The part that first lowers the queued distance
// counts the vertex for the next frontier, unless the first part of the round has (it then queued no distance).
__device__ __forceinline__ void sssp_pull_long(const SsspParams& p, const SsspPull& in, int fmin, unsigned L,
                                               unsigned G, unsigned* bits_next, int* best, unsigned long long& count,
                                               int& fnew, int lane, unsigned gwarp, unsigned nwarps) {
    const unsigned ntiles = (G + (1u << kPullTile) - 1u) >> kPullTile;
    if (ntiles > in.long_tiles || L > (unsigned)p.V) {
        if (lane == 0) atomicOr(&p.ctl->flags, C2G_FLAG_BOUNDS);
        return;
    }
    for (unsigned t = gwarp; t < ntiles; t += nwarps) {
        unsigned g0 = t << kPullTile;
        const unsigned g1 = min(g0 + (1u << kPullTile), G);
        for (unsigned o = (unsigned)ldcg(in.long_mark + t); g0 < g1 && o < L; o += 32) {
            const unsigned j = o + (unsigned)lane;
            unsigned base = 0x7fffffffu, next = 0xffffffffu;
            int v = 0, d = INT_MIN, bq = 0, i = 0;
            if (j < L) {
                const int2 ve = ldcg(p.q[0] + j);
                const long long at = __double_as_longlong(ldcg(in.long_at + j));
                v = ve.x;
                base = (unsigned)ve.y;
                next = j + 1 < L ? (unsigned)ldcg(p.q[0] + j + 1).y : G;
                bq = (int)(at >> 32);
                i = (int)(unsigned)at;
                d = ldcg(p.dist + v);
            }
            const unsigned stop = min(g1, (unsigned)__shfl_sync(kFull, (int)next, 31));
            best[lane] = d;
            __syncwarp();
            for (unsigned g = g0 + (unsigned)lane; g - (unsigned)lane < stop; g += 32u) {
                const int k = owner_lane(base, g);
                const int ki = __shfl_sync(kFull, i, k);
                const unsigned kb = (unsigned)__shfl_sync(kFull, (int)base, k);
                if (g < stop) {
                    const int bk = *(volatile int*)(best + k);
                    int unused;
                    const int nb = pull_group(in, p.dist, ki + 4 * (int)(g - kb), bk - fmin, bk, &unused);
                    if (nb < bk) atomicMin(best + k, nb);
                }
            }
            __syncwarp();
            const int nb = best[lane];
            __syncwarp();
            if (nb < d) {
                const int old = atomicMin(p.dist + v, nb);
                if (nb < old) {
                    fnew = min(fnew, nb);
                    const int deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
                    if (deg > 0) {
                        if (old == bq) count += (1ull << 32) | (unsigned)deg;
                        if (!in.always) atomicOr(bits_next + ((unsigned)v >> 5), 1u << (v & 31));
                    }
                }
            }
            g0 = stop;
        }
    }
}

// kKept: every round pulls, and the map has at most one word per warp (sssp_pull_kept).
template <bool kKept>
__global__ void __launch_bounds__(kBitsThreads, kBitsBlocksPerSm)
    sssp_rounds_persistent(const SsspParams p, const SsspPull in) {
    TraversalCtl* ctl = p.ctl;
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(&ctl->bar_count);
    grid_sync_init();
    int* flags = &ctl->flags;
    const int lane = threadIdx.x & 31;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nthreads = gridDim.x * blockDim.x;
    const unsigned gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const unsigned V = (unsigned)p.V;
    __shared__ StageSmemD sm;
    __shared__ RoundShare share;
    const int wib = threadIdx.x >> 5;
    WarpStage fst{sm.v0[wib], sm.d0[wib], nullptr, 0};               // lists (push rounds)
    WarpStage lst{sm.v0[wib], sm.d0[wib], nullptr, 0, sm.xd0[wib]};  // long rows (pull rounds)
    unsigned long long tph = globaltimer_ns();

    // Init: dis = INF (src/sssp/purn/Main.cu:144-156), empty maps.
    for (unsigned v = gtid; v < V; v += nthreads) p.dist[v] = kInfDist;
    if (!in.always)
        for (unsigned i = gtid; i < ((V + 31u) >> 5); i += nthreads) in.bits[0][i] = in.bits[1][i] = 0u;
    if (gtid == 0) {
        // fmin of round 1 is 0 (the source); the next rounds' start empty
        ctl->farmin[2] = ctl->farmin[0] = INT_MAX;
        ctl->seeds = p.n_seeds;
    }
    if (threadIdx.x == 0) share = RoundShare{0ull, INT_MAX};
    if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
    // Source and pruned-record seeds (src/sssp/purn/Main.cu:160-181) form round 1.
    const int s_row = __ldg(p.row + p.source), s_deg = __ldg(p.row + p.source + 1) - s_row;
    if (gtid == 0) atomicMin(p.dist + p.source, 0);
    for (unsigned i = gtid; i < (unsigned)p.n_seeds; i += nthreads) atomicMin(p.dist + p.seed_v[i], p.seed_w[i]);
    if (!in.always) {
        if (gtid == 0) atomicOr(in.bits[1] + ((unsigned)p.source >> 5), 1u << (p.source & 31));
        for (unsigned i = gtid; i < (unsigned)p.n_seeds; i += nthreads) {
            const int v = p.seed_v[i];
            atomicOr(in.bits[1] + ((unsigned)v >> 5), 1u << (v & 31));
        }
    } else {
        // Pulls only: no list will hold the source's out-edges, so they are relaxed here
        // (most of a skewed graph is then one pull away); round 1 counts the same frontier.
        for (unsigned i = gtid; i < (unsigned)s_deg; i += nthreads) {
            const int2 ew = __ldg(p.adj + s_row + (int)i);
            atomicMin(p.dist + ew.x, ew.y);
        }
        unsigned long long c = gtid == 0 && s_deg > 0 ? (1ull << 32) | (unsigned)s_deg : 0ull;
        for (unsigned i = gtid; i < (unsigned)p.n_seeds; i += nthreads) {
            const int v = p.seed_v[i], deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
            if (deg > 0) c += (1ull << 32) | (unsigned)deg;
        }
        if (c) atomicAdd(&ctl->pcount[1], c);
    }
    if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
    phase_mark(ctl->phase_ns, tph, 0);

    extern __shared__ int4 kept_smem[];
    KeptWord* const kept = reinterpret_cast<KeptWord*>(kept_smem) + wib;  // kKept
    if (kKept) kept_load(p, in, *kept, lane, wib);
    int kept_b = 0;
    bool kept_stale = true;

    int cur = 1, iters = 0;
    bool counted = in.always != 0;  // this round's frontier is counted (a pull made it), not listed
    // kKept: the coming round's count and smallest frontier distance, loaded together after each barrier
    unsigned long long next_count = kKept ? ldcg(&ctl->pcount[1]) : 0ull;
    int next_fmin = kKept ? ldcg(&ctl->farmin[1]) : 0;
    for (;;) {
        const int buf = cur & 1, slot = cur % 3, nslot = (cur + 1) % 3, fslot = (cur + 2) % 3;
        unsigned long long c = kKept ? next_count : counted ? ldcg(&ctl->pcount[slot]) : 0ull;
        if (gtid == 0) ctl->qctr[nslot] = 0ull;
        if (!kKept && (!counted || (c != 0ull && (unsigned)c <= in.pull_min))) {
            bits_sweep(p, in.bits[buf], sssp_out(p, buf, slot), fst, gwarp, nwarps, lane);
            if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
            phase_mark(ctl->phase_ns, tph, 1);
            c = ldcg(&ctl->qctr[slot]);
        }
        const unsigned F = (unsigned)(c >> 32), T = (unsigned)c;
        if (F == 0) break;
        if (++iters > p.max_iter) {
            if (gtid == 0) atomicOr(flags, C2G_FLAG_ITER_CAP);
            break;
        }
        if (gtid == 0) {
            ctl->popped += F;
            ctl->relaxed += T;
            ctl->pcount[fslot] = 0ull;
            ctl->farmin[fslot] = INT_MAX;
            ctl->lctr[buf ^ 1] = 0ull;
        }
        unsigned long long count = 0ull;
        int fnew = INT_MAX;
        const bool pull = kKept || T > in.pull_min;  // grid-uniform
        const int fmin = kKept ? next_fmin : ldcg(&ctl->farmin[slot]);
        if (kKept) {
            sssp_pull_kept(p, in, fmin, *kept, kept_b, kept_stale, sm.v1[wib], lst, pull_long_out(p, in, buf), count, fnew,
                           lane, wib);
        } else if (pull) {
            sssp_pull(p, in, fmin, in.bits[buf], in.bits[buf ^ 1], sm.v1[wib], lst, pull_long_out(p, in, buf), count,
                      fnew, lane, wib);
        } else {
            constexpr int U = kSsspUnroll;
            unsigned* bits = in.bits[buf ^ 1];
            walk_frontier_edges<U>(
                p.q[buf], p.mark[buf], p.row, F, T, p.log_tile, p.mark_cap, V, p.E, flags,
                [&](int v, unsigned) { return ldcg(p.dist + v); },  // the owner's current distance
                [&](const bool* ok, const unsigned* idx, const int* du) {
                    int c2[U], nd[U], cd[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int2 ew = ok[u] ? __ldg(p.adj + idx[u]) : make_int2(0, 0);
                        c2[u] = ew.x;
                        nd[u] = du[u] + ew.y;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) cd[u] = ok[u] ? ldcg(p.dist + c2[u]) : INT_MIN;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (nd[u] < cd[u]) {  // an L2 read guards the update
                            atomicMin(p.dist + c2[u], nd[u]);
                            atomicOr(bits + ((unsigned)c2[u] >> 5), 1u << (c2[u] & 31));
                            fnew = min(fnew, nd[u]);
                        }
                    }
                },
                kBitsDynTiles ? &ctl->tilectr[slot] : nullptr);
        }
        round_totals(ctl, nslot, &share, count, fnew, lane);
        if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
        if (pull) {
            const unsigned long long lc = ldcg(&ctl->lctr[buf]);  // grid-uniform
            if (kKept) {
                next_count = ldcg(&ctl->pcount[nslot]);
                next_fmin = ldcg(&ctl->farmin[nslot]);
            }
            if (lc) {
                count = 0ull;
                fnew = INT_MAX;
                sssp_pull_long(p, in, fmin, (unsigned)(lc >> 32), (unsigned)lc, in.bits[buf ^ 1], sm.v1[wib], count,
                               fnew, lane, gwarp, nwarps);
                round_totals(ctl, nslot, &share, count, fnew, lane);
                if (!grid_sync(bar, flags, p.barrier_ns, p.bar_extra)) return;
                if (kKept) {
                    next_count = ldcg(&ctl->pcount[nslot]);
                    next_fmin = ldcg(&ctl->farmin[nslot]);
                }
            }
        }
        phase_mark(ctl->phase_ns, tph, 2);
        counted = pull;
        ++cur;
    }
    if (gtid == 0) ctl->iterations = iters;
}

// ---------------------------------------------------------------------------------------
// host side

constexpr size_t kKeptSmem = sizeof(KeptWord) * (kBitsThreads / 32);

static int sssp_geometry(c2g_graph* g) {
    if (g->geom_sssp.blocks > 0) return C2G_OK;
    int coop = 0;
    C2G_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g->device));
    if (!coop) return fail(C2G_ERR_UNSUPPORTED, "device %d lacks cooperative launch", g->device);
    int per_sm_a = 0, per_sm_b = 0, per_sm_c = 0;
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_a, sssp_persistent<false>, 512, 0));
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_b, sssp_persistent<true>, 512, 0));
    C2G_CUDA(cudaFuncSetAttribute(sssp_rounds_persistent<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kKeptSmem));
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_c, sssp_rounds_persistent<false>, kBitsThreads, 0));
    int per_sm_d = 0;
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_d, sssp_rounds_persistent<true>, kBitsThreads, kKeptSmem));
    per_sm_c = std::min(per_sm_c, per_sm_d);
    const int per_sm = per_sm_a < per_sm_b ? per_sm_a : per_sm_b;
    if (per_sm < 1 || per_sm_c < 1) return fail(C2G_ERR_CUDA, "SSSP kernel cannot be resident (occupancy 0)");
    g->geom_sssp.blocks = per_sm * g->num_sms;
    g->geom_sssp.threads = 512;
    g->geom_bits.blocks = per_sm_c * g->num_sms;
    g->geom_bits.threads = kBitsThreads;
    return C2G_OK;
}

void sssp_free(c2g_graph* g) {
    SsspWork& w = g->sssp;
    void* ptrs[] = {w.dist, w.stamp, w.farstamp, w.q[0], w.q[1], w.mark[0], w.mark[1],
                    w.far, w.pull_mark, w.bits, w.ctl, w.st};
    for (void* ptr : ptrs)
        if (ptr) cudaFree(ptr);
    w = SsspWork();
}

static int pull_mark_alloc(c2g_graph* g) {
    C2G_CUDA(cudaMalloc(&g->sssp.pull_mark, sizeof(int) * ((size_t)(g->in_edges >> (kPullTile + 2)) + 2)));
    return C2G_OK;
}

static int sssp_alloc(c2g_graph* g) {
    SsspWork& w = g->sssp;
    const int log_tile = g->sssp_cfg.log_tile;
    if (w.dist && w.log_tile == log_tile) {
        if (g->in_adj && !w.pull_mark) return pull_mark_alloc(g);
        return C2G_OK;
    }
    if (w.dist) sssp_free(g);
    const size_t V = (size_t)g->V;
    const size_t nv = V ? V : 1;
    const unsigned mark_cap = (unsigned)(((size_t)g->E >> log_tile) + 2);
    C2G_CUDA(cudaMalloc(&w.dist, sizeof(int) * nv));
    C2G_CUDA(cudaMalloc(&w.stamp, sizeof(int) * nv));
    C2G_CUDA(cudaMalloc(&w.farstamp, sizeof(int) * nv));
    for (int b = 0; b < 2; ++b) {
        C2G_CUDA(cudaMalloc(&w.q[b], sizeof(int2) * nv));
        C2G_CUDA(cudaMalloc(&w.mark[b], sizeof(int) * mark_cap));
    }
    C2G_CUDA(cudaMalloc(&w.far, sizeof(int) * nv * 3));
    C2G_CUDA(cudaMalloc(&w.bits, sizeof(unsigned) * 2 * ((nv + 31) / 32)));
    int rc;
    if (g->in_adj && (rc = pull_mark_alloc(g))) return rc;
    C2G_CUDA(cudaMalloc(&w.ctl, sizeof(TraversalCtl)));
    C2G_CUDA(cudaMalloc(&w.st, sizeof(StampState)));
    C2G_CUDA(cudaMemsetAsync(w.stamp, 0xff, sizeof(int) * nv, g->stream));
    C2G_CUDA(cudaMemsetAsync(w.farstamp, 0xff, sizeof(int) * nv, g->stream));
    C2G_CUDA(cudaMemsetAsync(w.st, 0, sizeof(StampState), g->stream));
    w.mark_cap = mark_cap;
    w.log_tile = log_tile;
    return C2G_OK;
}

// Round rule of a launch.  A pull's cost is its pass over the vertices (80 - 110 us at 4.2M),
// a push's its frontier's out-edges (150 us for 15.6M of 65M) and a second barrier.
//   * kPullDiv: a round pulls when its frontier holds more than 1/4 of the edges (scale 22:
//     1.05 ms a query, at 1/10 1.17 ms: the first pull meets rows that nothing has reached).
//   * kPullAlways*: below these sizes a whole pull is about as short as a barrier (3.5 - 5 us
//     once most rows are pruned), so every round pulls, without map, list or second barrier
//     (scale 16, 1M edges: 134 us against 250 us with push rounds; scale 12: 89 against 120).
//     The vertex bound keeps graphs of few edges and very many rounds on sparse pushes.
//   * kPullMaxDegree: a warp pulls 32 vertices; with few vertices and very long rows too few
//     warps would have work.
constexpr int64_t kPullMaxDegree = 128;
constexpr int64_t kPullDiv = 4;
constexpr int64_t kPullAlwaysEdges = 4000000;
constexpr int32_t kPullAlwaysVertices = 300000;

static void sssp_round_rule(const c2g_graph* g, SsspPull& in) {
    const SsspWork& w = g->sssp;
    const size_t nw = ((size_t)g->V + 31) / 32;
    in.row = g->in_row;
    in.adj = g->in_adj;
    in.shift = g->in_shift;
    in.bits[0] = w.bits;
    in.bits[1] = w.bits + nw;
    in.long_at = reinterpret_cast<double*>(w.far);  // the far piles belong to delta > 0
    in.long_mark = w.pull_mark;
    in.long_tiles = w.pull_mark ? (unsigned)((g->in_edges >> (kPullTile + 2)) + 2) : 0u;
    in.pull_min = ~0u;
    in.always = 0;
    if (!g->in_adj || g->hw_negative || g->E > kPullMaxDegree * (int64_t)g->V) return;
    in.always = g->E <= kPullAlwaysEdges && g->V <= kPullAlwaysVertices;
    in.pull_min = in.always ? 0u : (unsigned)(g->E / kPullDiv);
}

int sssp_launch(c2g_graph* g, int32_t source, const int32_t* seed_v, const int32_t* seed_w, int32_t n_seeds,
                int32_t* dist_dev, float* ms) {
    int rc;
    if ((rc = sssp_geometry(g))) return rc;
    if (g->sssp_cfg.delta == 0 && (rc = ensure_in_rows(g))) return rc;
    if ((rc = sssp_alloc(g))) return rc;
    if (!g->adj_w) return fail(C2G_ERR_UNSUPPORTED, "graph has no int32 weights (wlist)");
    SsspWork& w = g->sssp;
    SsspParams p;
    p.row = g->row;
    p.adj = g->adj_w;
    p.V = g->V;
    p.E = (unsigned)g->E;
    p.dist = dist_dev ? dist_dev : w.dist;
    p.stamp = w.stamp;
    p.farstamp = w.farstamp;
    p.stamp_extent = g->V;
    p.q[0] = w.q[0];
    p.q[1] = w.q[1];
    p.mark[0] = w.mark[0];
    p.mark[1] = w.mark[1];
    const size_t nv = g->V ? (size_t)g->V : 1;
    p.far[0] = w.far;
    p.far[1] = w.far + nv;
    p.far[2] = w.far + 2 * nv;
    p.ctl = w.ctl;
    p.st = w.st;
    p.source = source;
    p.seed_v = seed_v;
    p.seed_w = seed_w;
    p.n_seeds = n_seeds;
    p.delta = g->sssp_cfg.delta;
    p.log_tile = w.log_tile;
    p.max_iter = g->sssp_cfg.max_iter;
    p.mark_cap = w.mark_cap;
    p.barrier_ns = g->barrier_ns ? g->barrier_ns : 2000000000ull;
    p.bar_extra = g->stall_next_sssp ? 1u : 0u;
    g->stall_next_sssp = 0;
    C2G_CUDA(cudaMemsetAsync(w.ctl, 0, sizeof(TraversalCtl), g->stream));
    const bool delta = p.delta > 0;
    SsspPull in;
    sssp_round_rule(g, in);
    // delta = 0: Bellman-Ford rounds; delta > 0: near/far buckets
    void* args[] = {&p, &in};
    const int words = (g->V + 31) / 32, warps = kBitsThreads / 32;
    const int blocks = delta ? g->geom_sssp.blocks
                     : in.always ? std::min(g->geom_bits.blocks, (words + warps - 1) / warps)
                                 : g->geom_bits.blocks;
    const bool kept = !delta && in.always && words <= blocks * warps;
    C2G_CUDA(cudaEventRecord(g->ev0, g->stream));
    C2G_CUDA(cudaLaunchCooperativeKernel(delta  ? (const void*)sssp_persistent<true>
                                         : kept ? (const void*)sssp_rounds_persistent<true>
                                                : (const void*)sssp_rounds_persistent<false>,
                                         dim3(blocks),
                                         dim3(delta ? g->geom_sssp.threads : g->geom_bits.threads), args, kept ? kKeptSmem : 0,
                                         g->stream));
    C2G_CUDA(cudaEventRecord(g->ev1, g->stream));
    if (ms) {
        C2G_CUDA(cudaEventSynchronize(g->ev1));
        C2G_CUDA(cudaEventElapsedTime(ms, g->ev0, g->ev1));
    }
    return C2G_OK;
}

}  // namespace c2g

// ---------------------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some callers cannot let this library allocate device memory per call.  Examples are a
// host whose device memory is owned entirely by another allocator, and a serving loop
// that must not call cudaMalloc/cudaFree after start-up (both may synchronise the device
// and stall every stream).  c2g_sssp_noalloc runs the same single-query kernel as
// c2g_sssp on arrays the caller already holds on the device.  Its scratch memory
// (round tags, frontier queues, tile markers and the launch control block) is
// g_sssp_noalloc_scratch below: a fixed array, loaded with the library on every GPU that
// uses it and held until the process exits.  Its size bounds the graphs this entry
// point accepts (C2G_NOALLOC_MAX_V vertices, C2G_NOALLOC_MAX_E edges).

namespace c2g {
namespace {

constexpr int kNoAllocLogTile = 8;
constexpr size_t kNoAllocMarks = ((size_t)C2G_NOALLOC_MAX_E >> kNoAllocLogTile) + 2;

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffStamp = 0;
constexpr size_t kOffFarstamp = kOffStamp + align256(sizeof(int) * (size_t)C2G_NOALLOC_MAX_V);
constexpr size_t kOffQ0 = kOffFarstamp + align256(sizeof(int) * (size_t)C2G_NOALLOC_MAX_V);
constexpr size_t kOffQ1 = kOffQ0 + align256(sizeof(int2) * (size_t)C2G_NOALLOC_MAX_V);
constexpr size_t kOffMark0 = kOffQ1 + align256(sizeof(int2) * (size_t)C2G_NOALLOC_MAX_V);
constexpr size_t kOffMark1 = kOffMark0 + align256(sizeof(int) * kNoAllocMarks);
constexpr size_t kOffCtl = kOffMark1 + align256(sizeof(int) * kNoAllocMarks);
constexpr size_t kOffSt = kOffCtl + align256(sizeof(TraversalCtl));
constexpr size_t kNoAllocScratchBytes = kOffSt + align256(sizeof(StampState));

constexpr int kNoAllocMaxDevices = 64;
void* g_noalloc_base[kNoAllocMaxDevices];  // device address of the scratch, per device (null: not looked up)
std::mutex g_noalloc_mu;

}  // namespace

// The scratch.  Zero at module load: round tags start above 0 and the tag bases start at
// 0, so no clearing is needed before the first call; the control block is cleared on the
// caller's stream before every launch.
static __device__ __align__(256) unsigned char g_sssp_noalloc_scratch[kNoAllocScratchBytes];

}  // namespace c2g

extern "C" int c2g_sssp_noalloc(const int32_t* row, const void* adj, int32_t V, int64_t E, int32_t source,
                                int32_t* dist, void* stream, c2g_stats* stats) {
    using namespace c2g;
    if (!row || !adj || !dist) return fail(C2G_ERR_ARG, "noalloc SSSP: NULL argument");
    if (V < 1 || V > C2G_NOALLOC_MAX_V)
        return fail(C2G_ERR_RANGE, "noalloc SSSP: V = %d outside [1, %d] (size of the static scratch)", V,
                    C2G_NOALLOC_MAX_V);
    if (E < 0 || E > C2G_NOALLOC_MAX_E)
        return fail(C2G_ERR_RANGE, "noalloc SSSP: E = %lld outside [0, %lld] (size of the static scratch)",
                    (long long)E, (long long)C2G_NOALLOC_MAX_E);
    if (source < 0 || source >= V) return fail(C2G_ERR_RANGE, "source %d out of range [0,%d)", source, V);
    int dev = 0;
    C2G_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(C2G_ERR_UNSUPPORTED, "device index %d too large", dev);
    // Once per device, with that device current: the device address of the scratch.
    // The host-side name of a __device__ array is not a device address.  Only a
    // successful lookup is kept; a failed one (say, made during a stream capture) is
    // retried by the next call.
    unsigned char* base = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_base[dev]) {
            void* addr = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&addr, g_sssp_noalloc_scratch);
            if (e != cudaSuccess) {
                cudaGetLastError();
                return fail(C2G_ERR_CUDA, "noalloc SSSP: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            }
            g_noalloc_base[dev] = addr;
        }
        base = static_cast<unsigned char*>(g_noalloc_base[dev]);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    int coop = 0, per_sm = 0, sms = 0;
    C2G_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return fail(C2G_ERR_UNSUPPORTED, "device %d lacks cooperative launch", dev);
    C2G_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sssp_persistent<false>, 512, 0));
    if (per_sm < 1) return fail(C2G_ERR_CUDA, "SSSP kernel cannot be resident (occupancy 0)");

    SsspParams p;
    p.row = row;
    p.adj = static_cast<const int2*>(adj);
    p.E = (unsigned)E;
    p.V = V;
    p.dist = dist;
    p.stamp = reinterpret_cast<int*>(base + kOffStamp);
    p.farstamp = reinterpret_cast<int*>(base + kOffFarstamp);
    p.stamp_extent = C2G_NOALLOC_MAX_V;  // the array serves graphs of every size
    p.q[0] = reinterpret_cast<int2*>(base + kOffQ0);
    p.q[1] = reinterpret_cast<int2*>(base + kOffQ1);
    p.mark[0] = reinterpret_cast<int*>(base + kOffMark0);
    p.mark[1] = reinterpret_cast<int*>(base + kOffMark1);
    p.far[0] = p.far[1] = p.far[2] = nullptr;  // the near/far split is off here
    p.ctl = reinterpret_cast<TraversalCtl*>(base + kOffCtl);
    p.st = reinterpret_cast<StampState*>(base + kOffSt);
    p.source = source;
    p.seed_v = nullptr;
    p.seed_w = nullptr;
    p.n_seeds = 0;
    p.delta = 0;
    p.log_tile = kNoAllocLogTile;
    p.max_iter = 1 << 20;
    p.mark_cap = (unsigned)(((size_t)E >> kNoAllocLogTile) + 2);
    p.barrier_ns = 2000000000ull;
    p.bar_extra = 0u;
    C2G_CUDA(cudaMemsetAsync(p.ctl, 0, sizeof(TraversalCtl), s));
    void* args[] = {&p};
    C2G_CUDA(cudaLaunchCooperativeKernel((const void*)sssp_persistent<false>, dim3(per_sm * sms), dim3(512), args, 0,
                                         s));
    TraversalCtl ctl;
    C2G_CUDA(cudaMemcpyAsync(&ctl, p.ctl, sizeof(ctl), cudaMemcpyDeviceToHost, s));
    C2G_CUDA(cudaStreamSynchronize(s));
    if (ctl.flags & (C2G_FLAG_BARRIER_TIMEOUT | C2G_FLAG_QUEUE_OVERFLOW | C2G_FLAG_BOUNDS)) {
        static const StampState reset{1 << 30, 1 << 30, {0, 0}};
        cudaMemcpyAsync(p.st, &reset, sizeof(reset), cudaMemcpyHostToDevice, s);
        cudaStreamSynchronize(s);
    }
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->source = source;
        stats->iterations = ctl.iterations;
        stats->vertices_popped = ctl.popped;
        stats->edges_relaxed = ctl.relaxed;
        stats->status_flags = ctl.flags;
        stats->alg_bytes = 4.0 * V + 16.0 * (double)ctl.popped + 12.0 * (double)ctl.relaxed;
    }
    if (ctl.flags & C2G_FLAG_BARRIER_TIMEOUT) return fail(C2G_ERR_TIMEOUT, "grid barrier wait ran out");
    if (ctl.flags & (C2G_FLAG_QUEUE_OVERFLOW | C2G_FLAG_BOUNDS))
        return fail(C2G_ERR_OVERFLOW, "device queue or index check failed");
    return C2G_OK;
}
