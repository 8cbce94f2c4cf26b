// Batched multi-query SSSP for sm_103a: up to thousands of sources in ONE persistent
// cooperative launch, with per-query bitmask frontiers.
//
// The reference runs one query per launch (src/sssp/purn/Main.cu:67-99) and, in its
// PM mode, two queries on two streams (src/sssp/purn-perk/Main.cu:51-53,107,164).  Here
// Q queries (padded to a multiple of 32) share every pass over the graph:
//   * state is vertex-major: dist[v][Q] int32, so the 32 queries of one "word" w of a
//     vertex occupy one 128-byte line;
//   * a frontier entry is a (vertex, word) pair with a 32-bit mask of the word's queries
//     that improved the vertex in the previous round;
//   * expansion: a warp reads 32 edges of an entry (one per lane) and broadcasts them;
//     for each edge every lane relaxes one query of the word with one coalesced
//     128-byte read of the target's row, so an edge read from HBM serves all active
//     queries of its word;
//   * an improvement is red.min on the distance and red.or of the query bits into the
//     target's (vertex, word) mask: nothing on the relaxation path waits for an atomic;
//   * a round is two phases: a sweep of the mask words that builds the frontier (with
//     edge-base prefix and tile markers), then the expansion.
// Results are the same int32 fixed points as one c2g_sssp call per source.
#include <climits>
#include <cmath>
#include <cstring>
#include <algorithm>
#include <vector>

#include "device_common.cuh"
#include "f32x2.h"
#include "fp64_mul.h"
#include "internal.h"

namespace c2g {

struct BatchParams {
    const int* row;
    const int2* adj;
    unsigned E;
    int V;
    int logW;  // words per vertex = 1 << logW
    int Q;     // padded query count = 32 << logW
    int nq;    // real queries (a resident batch: slots up to the last running one)
    unsigned live[32];  // of those, by query word: the queries (slots) at work
    int* dist;          // [V][Q]
    unsigned* mask;     // [V][W] next-round masks
    int2* q[2];         // entries (v*W + w, edge base)
    unsigned* qmask[2]; // gathered masks per entry
    int* mark[2];
    TraversalCtl* ctl;
    const int* sources;   // [nq]
    const int* seed_off;  // [nq+1] offsets into seed_v/seed_w (or nullptr)
    const int* seed_v;
    const int* seed_w;
    unsigned qcap;
    unsigned mark_cap;
    int max_iter;
    unsigned long long barrier_ns;
    long long* counters;  // [2]: relaxations (query, edge), edge-word steps
    int tile_big_log;     // log2 of the big tile's edge-word steps (>= kBatchTileLog)
    int tile_min_log;     // a round walks big tiles when it has >= 2^tile_min_log of them per warp
    int epoch_rounds;     // > 0: an epoch of a resident batch (no initialisation; at most this many rounds)
    RoundTrace* trace;    // [kMaxTraceRounds + 1] per-round trace
    // pull rounds: in-edge rows ordered by weight (in_edges.cu); a round pulls when its
    // (query, edge) relaxations exceed pull_min (~0: never); amask[b] holds the frontier's lanes per
    // (vertex, word) of the rounds of parity b (zero elsewhere); qmin the smallest distance that
    // entered each query's frontier, by round slot
    const int* in_row;
    const int2* in_adj;
    const int2* in_seg;
    unsigned in_segs;
    int in_shift;
    unsigned long long pull_min;
    unsigned long long pull_next;  // the same, once a round of the launch has pulled (batches of one or two words)
    unsigned pull_groups;          // groups of WP query words with queries
    unsigned* amask[2];
    int* qmin;  // [3][Q]
};

// Warp tiles of the expansion: markers are laid every 2^kBatchTileLog edge-word steps; a
// round with enough work (at least 2^tile_min_log big tiles per warp) walks tiles of
// 2^tile_big_log steps (every 2^(big - kBatchTileLog)-th marker), a smaller one tiles of
// 2^kBatchTileLog.  The handle's defaults are big 512, at least 16 per warp (256 sources
// at scale 22: 132 ms per SSSP batch with 128-step tiles, 121 ms with 512; 32 sources at
// scale 20: 4.6 ms with 128, 5.4 ms with 512, too few tiles per warp);
// c2g_sssp_batch_autotune picks them per batch.
constexpr int kBatchTileLog = 7;

__device__ __forceinline__ int batch_tile_log(unsigned T, unsigned nwarps, int big, int min_log) {
    return big > kBatchTileLog && (unsigned long long)T >= ((unsigned long long)nwarps << (big + min_log))
               ? big
               : kBatchTileLog;
}

// The batched push walks big tiles of 512 steps in rounds with at least 16 per warp.
constexpr int kPushTileBig = 9;
constexpr int kPushTileMin = 4;

__device__ __forceinline__ void trace_round(RoundTrace* tr, int i, long long work, int shape) {
    if (i <= kMaxTraceRounds) tr[i] = RoundTrace{globaltimer_ns(), work, shape, 0u};
}

// The end of round i's first phase (right after its grid barrier).
__device__ __forceinline__ void trace_mid(RoundTrace* tr, int i) {
    if (i >= 0 && i <= kMaxTraceRounds) tr[i].mid_ns = (unsigned)(globaltimer_ns() - tr[i].t_ns);
}

__device__ __forceinline__ FrontierOut batch_out(const BatchParams& p, int buf, int slot) {
    FrontierOut o;
    o.q = p.q[buf];
    o.val = reinterpret_cast<float*>(p.qmask[buf]);  // mask bits travel in the value slot
    o.mark = p.mark[buf];
    o.ctr = &p.ctl->qctr[slot];
    o.cap = p.qcap;
    o.mark_cap = p.mark_cap;
    o.log_tile = kBatchTileLog;
    o.flags = &p.ctl->flags;
    return o;
}

// Build a round's frontier from the improvement masks: a sweep over all (vertex, word)
// mask words; each non-zero word is cleared and, when the vertex has out-edges, becomes an
// entry (v * W + w, edge base) carrying the mask.  Entries come out in sweep order per
// warp.  Relaxations set masks with fire-and-forget red.or, so no relaxation waits on an
// atomic's return; the sweep reads V * W words per round.
// Late rounds leave most words empty: one block of 32 words at a time, a sweep was a chain of loads (0.12
// ms a round of 256 queries at scale 22, 0.035 with 4; of a whole query batch's 42.1 ms 4.8, now 3.1; 2
// blocks 3.6, 8 3.4).
constexpr int kSweepBlocks = 4;  // blocks of 32 mask words a warp reads at once

__device__ __forceinline__ void batch_sweep(const BatchParams& p, const FrontierOut& out, unsigned* am,
                                            unsigned long long* pcount, WarpStage& fst, unsigned gwarp,
                                            unsigned nwarps, int lane) {
    const unsigned nm = (unsigned)p.V << p.logW;
    unsigned long long rel = 0;  // (query, edge) relaxations of the frontier
    for (unsigned b = gwarp * 32u * kSweepBlocks; b < nm; b += nwarps * 32u * kSweepBlocks) {
        unsigned m[kSweepBlocks];
        int deg[kSweepBlocks];
#pragma unroll
        for (int u = 0; u < kSweepBlocks; ++u) {
            const unsigned i = b + 32u * u + (unsigned)lane;
            m[u] = i < nm ? ldcg(p.mask + i) : 0u;
        }
        unsigned any = 0u;
#pragma unroll
        for (int u = 0; u < kSweepBlocks; ++u) any |= m[u];
        if (!__any_sync(kFull, any != 0u)) continue;
#pragma unroll
        for (int u = 0; u < kSweepBlocks; ++u) {
            const unsigned i = b + 32u * u + (unsigned)lane;
            deg[u] = 0;
            if (m[u]) {
                p.mask[i] = 0u;
                const int v = (int)(i >> p.logW);
                deg[u] = __ldg(p.row + v + 1) - __ldg(p.row + v);
            }
        }
#pragma unroll
        for (int u = 0; u < kSweepBlocks; ++u) {
            const unsigned i = b + 32u * u + (unsigned)lane;
            if (am && m[u] != 0u && deg[u] > 0) {
                am[i] = m[u];  // the pull rounds' lookup of the frontier's lanes
                rel += (unsigned long long)__popc(m[u]) * (unsigned long long)deg[u];
            }
            stage_push(fst, out, m[u] != 0u && deg[u] > 0, (int)i, deg[u], __int_as_float((int)m[u]));
        }
    }
    stage_flush(fst, out);
    if (am) {
        for (int o = 16; o >= 1; o >>= 1) rel += __shfl_xor_sync(kFull, rel, o);
        if (lane == 0 && rel) atomicAdd(pcount, rel);
    }
}

constexpr int kBatchUnroll = 4;  // relaxation items in flight per lane
// Launch shape of the batched SSSP: 3 blocks of 384 threads per SM (36 warps) measured
// faster than 2 x 512 (32 warps) at the same 4 items per lane (132-135 vs 140 ms for 256
// sources at scale 22), 1 x 512 with 8-12 items (220 ms) and 6 x 256 (192 ms).
constexpr int kSsspBatchThreads = 384;
constexpr int kSsspBatchBlocksPerSm = 3;
constexpr int kQminCap = 1024;  // query slots whose frontier minima are tracked (more: taken as 0)

// Lane compaction of one owner run: the run's work is the items (edge ei, active-query
// slot j) for ei in [0, len) and j in [0, cnt), numbered i = ei * cnt + j; lane l takes
// items l, l + 32, l + 64, ... so every lane of a warp step relaxes something even when
// few of the word's 32 queries are active.  The (ei, j) of a lane advance by 32 items
// per step without a division (32 = dq * cnt + dr).  Lane 0 holds the lowest item, so
// the loop condition is warp-uniform; body(ei[U], j[U]) must check ei < len.
template <int U, typename Body>
__device__ __forceinline__ void owner_items(unsigned cnt, unsigned len, int lane, Body body) {
    const float rc = __frcp_rn((float)cnt);  // exact enough: (l + 0.5) / cnt is >= 1/64 from an integer
    int ei = (int)(((float)lane + 0.5f) * rc);
    int j = lane - ei * (int)cnt;
    const int dq = (int)(32.5f * rc);
    const int dr = 32 - dq * (int)cnt;
    while ((unsigned)__shfl_sync(kFull, ei, 0) < len) {
        int eis[U], js[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            eis[u] = ei;
            js[u] = j;
            ei += dq;
            j += dr;
            if (j >= (int)cnt) {
                j -= (int)cnt;
                ++ei;
            }
        }
        body(eis, js);
    }
}

// Pull round of the batched SSSP.  In a dense round (most (vertex, word) pairs improved in
// the previous round) the expansion reads a 128-byte distance line per edge-word step and
// issues red.min for every improvement.  A pull round reads in-edges instead: for each target
// v and query word it takes the minimum of dist[u] + w over the in-edges u -> v whose source
// improved in the previous round (amask), lane by lane (lane = query), and compares it with
// dist[v].  The rows are ordered by weight, and v's row ends for a group of 4 query words at the
// first edge whose weight is not below dist[v][q] - qmin[q] for any of its queries q (qmin: the
// smallest distance in q's frontier): no later edge can improve v.  Without that bound a
// pull read every live in-edge's lines, 11.3 ms per dense round of 256 queries at scale 22; most
// rows now end within their first 4 edges: 8.0, 4.6, then 3.0 - 2.1 ms (distances of 4.3 GB
// read once take 0.65).
//
// Items are (16 vertices, word group) and (4 segments of long rows, word group), in
// word-group-major order.  A warp stages the first 4 in-edges of the 16 rows and their
// sources' lanes (2 edges per lane, so 16 rows' loads are in flight together); a row that needs
// more is read on in chunks of 32 edges.  Rows of up to kInHead edges have one writer and get
// plain stores; longer rows are shared with their segments' warps and get atomics.  A row that
// few queries have reached needs all its edges: with 32 rows an item and 128 edges before the
// first segment, a warp that met 32 hubs took longer than the rest of the round (256 queries
// at scale 19: 15.0 ms a batch, now 8.3; at scale 22 44.8 and 44.3).
// Any order of relaxations reaches the same fixed point, so the distances are those of
// the push rounds; pull and push rounds mix freely.
//
// A warp holds 4 (row, word) slots at a time, lane = query: the 4 words of one row, or, with 1
// or 2 words per vertex (WP), 4 or 2 rows, so that narrow batches have as many lines in
// flight (31 queries on 685,230 vertices: 0.86 ms a round one row at a time, 0.42 ms four).
struct SPullChunk {  // shared memory of one warp
    int2* ed;        // [32] a chunk's live in-edges: source, weight
    uint4* mk;       // [32] and their sources' active lanes in the item's words
    int2* red;       // [16][4] first in-edges of 16 rows
    uint4* rmk;      // [16][4]
};

template <int WP>
__device__ __forceinline__ uint4 spull_lanes(const BatchParams& p, const unsigned* am, int u, unsigned w0) {
    const unsigned* ms = am + ((size_t)(unsigned)u << p.logW) + w0;
    if (WP == 4) return ldcg(reinterpret_cast<const uint4*>(ms));  // four words, 16-byte aligned
    return make_uint4(ldcg(ms), WP > 1 ? ldcg(ms + 1) : 0u, 0u, 0u);
}

__device__ __forceinline__ bool any_lane(const uint4& m) { return (m.x | m.y | m.z | m.w) != 0u; }
__device__ __forceinline__ unsigned word_of(const uint4& m, int j) {
    return j == 0 ? m.x : j == 1 ? m.y : j == 2 ? m.z : m.w;
}
__device__ __forceinline__ int bucket_floor(int w, int shift) { return (w >> shift) << shift; }

// Weights at or above the returned limit improve none of the warp's queries (cur: this lane's distances).
template <int WP>
__device__ __forceinline__ int spull_limit(const int* cur, const int* qm) {
    int m = cur[0] - qm[0];
#pragma unroll
    for (int j = 1; j < WP; ++j) m = max(m, cur[j] - qm[j]);
    return __reduce_max_sync(kFull, m);
}

// The source's distances of an in-edge (u, m: its active lanes), unreachable where inactive or !on.
template <int WP>
__device__ __forceinline__ void spull_line(const int* dist_w0, unsigned Qu, int u, const uint4& m, bool on, int lane,
                                           int* d) {
    const int* line = dist_w0 + (size_t)(unsigned)u * Qu;
#pragma unroll
    for (int j = 0; j < WP; ++j)  // L2-coherent: other warps lower distances during the round
        d[j] = on && ((word_of(m, j) >> lane) & 1u) ? ldcg(line + 32 * j) : kInfDist;
}

// In-edges [b, e) of a row, 32 at a time, as long as they are below its limit.
template <int WP>
__device__ __forceinline__ void spull_chunks(const BatchParams& p, const unsigned* am, const int* dist_w0, unsigned w0,
                                             const int* qm, int* cur, int lim, const SPullChunk& pc, int b, int e,
                                             int lane) {
    const unsigned Qu = (unsigned)p.Q;
    for (; b < e; b += 32) {
        int2 ed = make_int2(0, INT_MAX);
        if (b + lane < e) ed = __ldg(p.in_adj + b + lane);
        const unsigned below = __ballot_sync(kFull, bucket_floor(ed.y, p.in_shift) < lim);
        if (below == 0u) return;
        uint4 m = make_uint4(0u, 0u, 0u, 0u);
        if (ed.y < lim) m = spull_lanes<WP>(p, am, ed.x, w0);
        const bool live = any_lane(m);
        const unsigned lm = __ballot_sync(kFull, live);
        const unsigned n = (unsigned)__popc(lm);
        __syncwarp();  // the previous chunk's reads are done
        if (live) {
            const unsigned at = (unsigned)__popc(lm & ((1u << lane) - 1u));
            pc.ed[at] = ed;
            pc.mk[at] = m;
        }
        __syncwarp();
        for (unsigned k = 0; k < n; k += 2) {
            int d[2][WP], w[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned kk = k + h < n ? k + h : k;
                const int2 ek = pc.ed[kk];
                w[h] = ek.y;
                spull_line<WP>(dist_w0, Qu, ek.x, pc.mk[kk], ek.y < lim, lane, d[h]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int j = 0; j < WP; ++j) cur[j] = min(cur[j], d[h][j] + w[h]);
            if ((k & 7u) == 6u) lim = spull_limit<WP>(cur, qm);
        }
        lim = spull_limit<WP>(cur, qm);
        if (below != kFull) return;  // the chunk held the first edge beyond the limit
    }
}

// The improved lanes of target v's words, d0: its distances when the row was started.
template <int WP>
__device__ __forceinline__ void spull_store(const BatchParams& p, int v, unsigned w0, bool whole, const int* d0,
                                            const int* cur, int* qnew, int lane) {
#pragma unroll
    for (int j = 0; j < WP; ++j) {
        const bool imp = cur[j] < d0[j];
        const unsigned bits = __ballot_sync(kFull, imp);
        if (bits == 0u) continue;
        const size_t off = (size_t)(unsigned)v * (unsigned)p.Q + ((w0 + j) << 5) + lane;
        const unsigned vw = ((unsigned)v << p.logW) + w0 + (unsigned)j;
        if (imp) qnew[j] = min(qnew[j], cur[j]);
        if (whole) {  // this warp reads all of v's in-edges: no other writer
            if (imp) p.dist[off] = cur[j];
            if (lane == 0) p.mask[vw] = bits;
        } else {
            if (imp) atomicMin(p.dist + off, cur[j]);
            if (lane == 0) atomicOr(p.mask + vw, bits);
        }
    }
}

template <int WP>
__device__ __forceinline__ void sbatch_pull(const BatchParams& p, int buf, int slot, int nslot, unsigned* qctr,
                                            const SPullChunk& pc, int lane) {
    constexpr int RP = 4 / WP;  // rows at a time
    const unsigned Qu = (unsigned)p.Q;
    const unsigned nblk = ((unsigned)p.V + 15u) / 16u, per_group = nblk + (p.in_segs + 3u) / 4u;
    const unsigned nitems = WP == 4 ? per_group * p.pull_groups : per_group;
    const unsigned* am = p.amask[buf];
    unsigned w0 = ~0u;  // the word group of qm and qnew
    int qm[WP], qnew[WP];
    auto flush = [&]() {  // the group's smallest new distances join the next round's qmin
        if (w0 == ~0u) return;
#pragma unroll
        for (int j = 0; j < WP; ++j) {
            int* q = p.qmin + nslot * Qu + ((w0 + j) << 5) + lane;
            if (qnew[j] < ldcg(q)) atomicMin(q, qnew[j]);
        }
    };
    unsigned itn = next_tile(qctr, lane);
    for (unsigned it = itn; it < nitems; it = itn) {
        itn = next_tile(qctr, lane);  // the next item, fetched while this one runs
        const unsigned grp = (it / per_group) * 4u;
        if (grp != w0) {
            flush();
            w0 = grp;
#pragma unroll
            for (int j = 0; j < WP; ++j) {
                const unsigned q = ((w0 + j) << 5) + (unsigned)lane;
                // a query slot without a query never bounds a row
                qm[j] = q < (unsigned)p.nq ? ldcg(p.qmin + slot * Qu + q) : INT_MAX;
                qnew[j] = INT_MAX;
            }
        }
        const int* dist_w0 = p.dist + (w0 << 5) + lane;
        const unsigned k = it % per_group;
        if (k >= nblk) {
            // 4 segments: most hold no weight below their row's limit, so all limits are found first
            const unsigned s0 = (k - nblk) * 4u;
            int2 sg = make_int2(0, 0);
            int w = INT_MAX, se = 0;
            if (lane < 4 && s0 + lane < p.in_segs) {
                sg = __ldg(p.in_seg + s0 + lane);
                w = bucket_floor(__ldg(&p.in_adj[sg.y].y), p.in_shift);
                se = min(sg.y + kInSegment, __ldg(p.in_row + sg.x + 1));
            }
            int d[4][WP];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned v = (unsigned)__shfl_sync(kFull, sg.x, q);
#pragma unroll
                for (int j = 0; j < WP; ++j) d[q][j] = ldcg(dist_w0 + (size_t)v * Qu + 32 * j);
            }
            unsigned live = 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (__shfl_sync(kFull, w, q) < spull_limit<WP>(d[q], qm)) live |= 1u << q;
            while (live) {
                const int q = __ffs(live) - 1;
                live &= live - 1u;
                const int v = __shfl_sync(kFull, sg.x, q);
                int d0[WP], cur[WP];
#pragma unroll
                for (int j = 0; j < WP; ++j) cur[j] = d0[j] = ldcg(dist_w0 + (size_t)(unsigned)v * Qu + 32 * j);
                spull_chunks<WP>(p, am, dist_w0, w0, qm, cur, spull_limit<WP>(cur, qm), pc, __shfl_sync(kFull, sg.y, q),
                                 __shfl_sync(kFull, se, q), lane);
                spull_store<WP>(p, v, w0, false, d0, cur, qnew, lane);
            }
            continue;
        }
        const int v0 = (int)(k * 16u);
        int rs = 0, re = 0;
        if (lane < 16 && v0 + lane < p.V) {
            rs = __ldg(p.in_row + v0 + lane);
            re = __ldg(p.in_row + v0 + lane + 1);
        }
        unsigned todo = __ballot_sync(kFull, rs < re);
        if (todo == 0u) continue;
        // the first 4 in-edges of 16 rows, two per lane, and their sources' active lanes
        {
            const int row = lane >> 1;
            const int i = __shfl_sync(kFull, rs, row) + 2 * (lane & 1);
            __syncwarp();
            if ((todo >> row) & 1u) {
                const int4 x = __ldg(reinterpret_cast<const int4*>(p.in_adj + i));
                pc.red[2 * lane] = make_int2(x.x, x.y);
                pc.red[2 * lane + 1] = make_int2(x.z, x.w);
                const uint4 none = make_uint4(0u, 0u, 0u, 0u);  // the padding has no source
                pc.rmk[2 * lane] = x.y != INT_MAX ? spull_lanes<WP>(p, am, x.x, w0) : none;
                pc.rmk[2 * lane + 1] = x.w != INT_MAX ? spull_lanes<WP>(p, am, x.z, w0) : none;
            }
            __syncwarp();
        }
        while (todo) {
            int row[RP], d0[RP][WP], cur[RP][WP], lim[RP];
            bool valid[RP];
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                valid[r] = todo != 0u;  // warp-uniform
                row[r] = valid[r] ? __ffs(todo) - 1 : row[0];
                todo &= todo - 1u;
#pragma unroll
                for (int j = 0; j < WP; ++j)
                    cur[r][j] = d0[r][j] =
                        ldcg(dist_w0 + (size_t)(unsigned)(v0 + row[r]) * Qu + 32 * j);
            }
#pragma unroll
            for (int r = 0; r < RP; ++r) lim[r] = spull_limit<WP>(cur[r], qm);
#pragma unroll
            for (int h0 = 0; h0 < 4; h0 += 2) {  // two in-edges of each row in flight
                int d[2][RP][WP], w[2][RP];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int r = 0; r < RP; ++r) {
                        const int2 e = pc.red[4 * row[r] + h0 + h];
                        w[h][r] = e.y;
                        spull_line<WP>(dist_w0, Qu, e.x, pc.rmk[4 * row[r] + h0 + h], e.y < lim[r], lane, d[h][r]);
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int r = 0; r < RP; ++r)
#pragma unroll
                        for (int j = 0; j < WP; ++j)  // (the padding's weight is no summand)
                            if (d[h][r][j] != kInfDist) cur[r][j] = min(cur[r][j], d[h][r][j] + w[h][r]);
            }
            int pos[RP], end[RP];  // what is left of each row (of a long row's head)
            bool more = false;
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                const int vrs = __shfl_sync(kFull, rs, row[r]), vre = __shfl_sync(kFull, re, row[r]);
                pos[r] = vrs + 4;
                end[r] = min(vre, vrs + kInHead);
                if (!valid[r] || bucket_floor(pc.red[4 * row[r] + 3].y, p.in_shift) >= lim[r]) end[r] = pos[r];
                more |= pos[r] < end[r];
            }
            if (RP == 1) {
                if (more)
                    spull_chunks<WP>(p, am, dist_w0, w0, qm, cur[0], spull_limit<WP>(cur[0], qm), pc, pos[0],
                                     end[0], lane);
            } else {
                // the next 32 / RP in-edges of all rows at a time
                constexpr int EP = 32 / RP;
                while (more) {
#pragma unroll
                    for (int r = 0; r < RP; ++r) lim[r] = spull_limit<WP>(cur[r], qm);
                    int my_pos = pos[0], my_end = end[0], my_lim = lim[0];
#pragma unroll
                    for (int r = 1; r < RP; ++r)
                        if (lane / EP == r) {
                            my_pos = pos[r];
                            my_end = end[r];
                            my_lim = lim[r];
                        }
                    int2 ed = make_int2(0, INT_MAX);
                    if (my_pos + lane % EP < my_end) ed = __ldg(p.in_adj + my_pos + lane % EP);
                    const unsigned below = __ballot_sync(kFull, bucket_floor(ed.y, p.in_shift) < my_lim);
                    uint4 m = make_uint4(0u, 0u, 0u, 0u);
                    if (ed.y < my_lim) m = spull_lanes<WP>(p, am, ed.x, w0);
                    __syncwarp();  // the previous reads are done
                    pc.ed[lane] = ed;
                    pc.mk[lane] = m;
                    __syncwarp();
                    int n = 0;  // edges to read: up to the last one below its row's limit
#pragma unroll
                    for (int r = 0; r < RP; ++r)
                        n = max(n, 32 - __clz((int)((below >> (r * EP)) & ((1u << EP) - 1u))));
                    for (int h0 = 0; h0 < n; h0 += 2) {
                        int d[2][RP][WP], w[2][RP];
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int r = 0; r < RP; ++r) {
                                const int2 e = pc.ed[r * EP + h0 + h];
                                w[h][r] = e.y;
                                spull_line<WP>(dist_w0, Qu, e.x, pc.mk[r * EP + h0 + h], true, lane, d[h][r]);
                            }
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int r = 0; r < RP; ++r)
#pragma unroll
                                for (int j = 0; j < WP; ++j)
                                    if (d[h][r][j] != kInfDist) cur[r][j] = min(cur[r][j], d[h][r][j] + w[h][r]);
                    }
                    more = false;
#pragma unroll
                    for (int r = 0; r < RP; ++r) {
                        pos[r] += EP;
                        // a row goes on when all its staged edges were below the limit
                        if (((below >> (r * EP)) & ((1u << EP) - 1u)) != ((1u << EP) - 1u)) end[r] = pos[r];
                        more |= pos[r] < end[r];
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                if (!valid[r]) break;  // warp-uniform
                const int len = __shfl_sync(kFull, re, row[r]) - __shfl_sync(kFull, rs, row[r]);
                spull_store<WP>(p, v0 + row[r], w0, len <= kInHead, d0[r], cur[r], qnew, lane);
            }
        }
    }
    flush();
}

// WP: query words a pull takes at a time (1, 2, or 4 of four or more)
template <int WP>
__global__ void __launch_bounds__(kSsspBatchThreads, kSsspBatchBlocksPerSm) sssp_batch_persistent(const BatchParams p) {
    TraversalCtl* ctl = p.ctl;
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(&ctl->bar_count);
    grid_sync_init();
    int* flags = &ctl->flags;
    const int lane = threadIdx.x & 31;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nthreads = gridDim.x * blockDim.x;
    const unsigned gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const int W = 1 << p.logW;
    const unsigned Qu = (unsigned)p.Q;
    __shared__ __align__(16) StageSmemN<kSsspBatchThreads / 32> sm;
    const int wib = threadIdx.x >> 5;
    unsigned long long tph = globaltimer_ns();
    WarpStage fst{sm.v0[wib], sm.d0[wib], sm.x0[wib], 0};
    int* qtab = sm.v1[wib];  // slot -> query position table of the owner being expanded
    // pull rounds: in-edge chunks in the (empty) stage, 16 rows' first in-edges, new minima
    __shared__ uint4 rmk[kSsspBatchThreads / 32][64];
    __shared__ int qlow[kQminCap];
    const SPullChunk pc{reinterpret_cast<int2*>(sm.v0[wib]), reinterpret_cast<uint4*>(sm.d0[wib]),
                        reinterpret_cast<int2*>(sm.x0[wib]), rmk[wib]};
    const bool may_pull = p.pull_min != ~0ull, low = may_pull && p.Q <= kQminCap;
    if (may_pull && gtid < Qu) {
        // round 1: no distance is below 0 (seeds and weights are not negative); a slot without a query at work
        // bounds no row in any round (its distances may be anything)
        p.qmin[Qu + gtid] = !low || ((p.live[gtid >> 5] >> (gtid & 31u)) & 1u) ? 0 : INT_MAX;
        p.qmin[gtid] = p.qmin[2 * Qu + gtid] = low ? INT_MAX : 0;
    }
    if (low)
        for (unsigned q = threadIdx.x; q < Qu; q += blockDim.x) qlow[q] = INT_MAX;

    // An epoch of a resident batch starts from the state the previous epoch left: the
    // distances and the improvement masks (queries that joined since have their column
    // set and their source marked).
    if (p.epoch_rounds == 0) {
    // Init: dist = INF (vector stores), masks = 0.
    {
        const size_t n4 = ((size_t)p.V * (size_t)p.Q) >> 2;
        int4* d4 = reinterpret_cast<int4*>(p.dist);
        const int4 inf4 = make_int4(kInfDist, kInfDist, kInfDist, kInfDist);
        for (size_t i = gtid; i < n4; i += nthreads) d4[i] = inf4;
        const size_t nm = (size_t)p.V << p.logW;
        for (size_t i = gtid; i < nm; i += nthreads) p.mask[i] = 0u;
    }
    if (!grid_sync(bar, flags, p.barrier_ns)) return;

    // Sources and their seeds: dist[s][q] = 0, dist[seed][q] = min(w); mark them.  A warp
    // per query, its lanes over the seed records.
    for (unsigned qi = gwarp; qi < (unsigned)p.nq; qi += nwarps) {
        const int s = p.sources[qi];
        const unsigned bit = 1u << (qi & 31), w = qi >> 5;
        if (lane == 0) {
            atomicMin(p.dist + (size_t)s * p.Q + qi, 0);
            atomicOr(p.mask + ((size_t)s << p.logW) + w, bit);
        }
        if (p.seed_off)
            for (int k = p.seed_off[qi] + lane; k < p.seed_off[qi + 1]; k += 32) {
                atomicMin(p.dist + (size_t)p.seed_v[k] * p.Q + qi, p.seed_w[k]);
                atomicOr(p.mask + ((size_t)p.seed_v[k] << p.logW) + w, bit);
            }
    }
    if (!grid_sync(bar, flags, p.barrier_ns)) return;
    }
    phase_mark(ctl->phase_ns, tph, 0);

    long long relax = 0, steps = 0;
    int cur = 1, iters = 0;
    bool pulled = false;  // a round of this launch has pulled
    for (;;) {
        const int buf = cur & 1, slot = cur % 3;
        // Phase 1: this round's frontier from the masks of the previous one.
        if (gtid == 0) {
            ctl->qctr[(cur + 1) % 3] = 0ull;
            ctl->tilectr[(cur + 1) % 3] = 0u;
            ctl->pcount[(cur + 1) % 3] = 0ull;
        }
        batch_sweep(p, batch_out(p, buf, slot), may_pull ? p.amask[buf] : nullptr, &ctl->pcount[slot], fst, gwarp,
                    nwarps, lane);
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        phase_mark(ctl->phase_ns, tph, 1);
        const unsigned long long c = ldcg(&ctl->qctr[slot]);
        const unsigned F = (unsigned)(c >> 32), T = (unsigned)c;
        // pull when the frontier's (query, edge) relaxations exceed pull_min: the dense rounds
        // in which most active words have most of their queries active (the push pays a
        // red.min per improvement there), not every round with many edge-word steps
        const bool pull = ldcg(&ctl->pcount[slot]) > (WP < 4 && pulled ? p.pull_next : p.pull_min);  // grid-uniform
        pulled = pull || pulled;
        if (gtid == 0) trace_round(p.trace, iters, (long long)T, pull ? 1 : 0);
        if (F == 0) break;
        if (++iters > p.max_iter) {
            if (gtid == 0) atomicOr(flags, C2G_FLAG_ITER_CAP);
            break;
        }
        if (F > p.qcap || ((T + (1u << kBatchTileLog) - 1u) >> kBatchTileLog) > p.mark_cap) {
            if (gtid == 0) atomicOr(flags, C2G_FLAG_BOUNDS);
            break;
        }
        if (gtid == 0) {
            ctl->popped += F;
            ctl->relaxed += T;
        }

        if (may_pull) {
            // The previous round's frontier leaves the pull lookup (the lookup of this round,
            // amask[buf], is the one a pull reads; the next round writes amask[buf ^ 1]).
            const unsigned Fp = min((unsigned)(ldcg(&ctl->qctr[(cur + 2) % 3]) >> 32), p.qcap);
            for (unsigned j = gtid; j < Fp; j += nthreads) p.amask[buf ^ 1][ldcg(p.q[buf ^ 1] + j).x] = 0u;
            if (low && gtid < Qu) p.qmin[((cur + 2) % 3) * Qu + gtid] = INT_MAX;
        }
        if (pull) {
            if (gtid == 0) {
                steps += T;
                relax += (long long)ldcg(&ctl->pcount[slot]);
            }
            sbatch_pull<WP>(p, buf, slot, (cur + 1) % 3, &ctl->tilectr[slot], pc, lane);
        } else {
        // Phase 2: expand.  Warps take tiles of edge-word steps and walk owner runs: the
        // owner's row of distances is read once; its edges are read 32 at a time (one per
        // lane, coalesced) and broadcast by shuffles; each edge costs one 128-byte read of
        // the target's row for the 32 queries of the word, kBatchUnroll rows in flight.
        // Improvements are red.min on the distance and red.or on the target's mask.
        const int2* q = p.q[buf];
        const unsigned* qm = p.qmask[buf];
        const int* mark = p.mark[buf];
        const int tl = batch_tile_log(T, nwarps, p.tile_big_log, p.tile_min_log);
        const unsigned tile = 1u << tl;
        const unsigned ntiles = (T + tile - 1) >> tl;
        unsigned* tctr = &ctl->tilectr[slot];
        unsigned tn = next_tile(tctr, lane);
        for (unsigned t = tn; t < ntiles; t = tn) {
            tn = next_tile(tctr, lane);  // the next tile, fetched while this one runs
            unsigned e0 = t << tl;
            const unsigned e1 = min(e0 + tile, T);
            unsigned o = (unsigned)ldcg(mark + (t << (tl - kBatchTileLog)));
            while (e0 < e1) {
                const unsigned j = o + (unsigned)lane;
                unsigned base = 0x7fffffffu, endv = 0xffffffffu, msk = 0u, rs = 0u;
                int vw = 0;
                bool bad = false;
                if (j < F) {
                    const int2 qe = ldcg(q + j);
                    vw = qe.x;
                    base = (unsigned)qe.y;
                    const int v = vw >> p.logW;
                    rs = (unsigned)__ldg(p.row + v);
                    const unsigned deg = (unsigned)__ldg(p.row + v + 1) - rs;
                    endv = base + deg;
                    bad = rs + deg > p.E || deg == 0u;
                    msk = ldcg(qm + j);
                }
                const unsigned seg_end = min(e1, (unsigned)__shfl_sync(kFull, endv, 31));
                if (__any_sync(kFull, bad) || seg_end <= e0 || o >= F ||
                    (unsigned)__shfl_sync(kFull, (int)base, 0) > e0) {
                    if (lane == 0) atomicOr(flags, C2G_FLAG_BOUNDS);
                    break;
                }
                for (int k = 0; k < 32; ++k) {
                    const unsigned kb = (unsigned)__shfl_sync(kFull, (int)base, k);
                    if (kb >= seg_end) break;
                    const unsigned ke = (unsigned)__shfl_sync(kFull, (int)endv, k);
                    const unsigned lo = max(e0, kb), hi = min(seg_end, ke);
                    if (lo >= hi) continue;
                    const int kvw = __shfl_sync(kFull, vw, k);
                    const unsigned km = (unsigned)__shfl_sync(kFull, (int)msk, k);
                    const unsigned krs = (unsigned)__shfl_sync(kFull, (int)rs, k);
                    const unsigned w = (unsigned)kvw & (unsigned)(W - 1);
                    const unsigned cnt = (unsigned)__popc(km);
                    // slot -> query position of the word's active queries
                    if ((km >> lane) & 1u) qtab[__popc(km & ((1u << lane) - 1u))] = lane;
                    __syncwarp();
                    const int qp = (unsigned)lane < cnt ? qtab[lane] : 0;
                    __syncwarp();
                    int* dw = p.dist + (w << 5);  // + v * Q + query position
                    unsigned* mrow = p.mask + w;  // + (v << logW): mask word of v
                    // L2-coherent: the owner improved in the previous round.
                    const int du = (unsigned)lane < cnt ? ldcg(dw + (size_t)((unsigned)kvw >> p.logW) * Qu + qp) : 0;
                    const unsigned len = hi - lo;
                    const int2* eadj = p.adj + krs + (lo - kb);
                    owner_items<kBatchUnroll>(cnt, len, lane, [&](const int* eis, const int* js) {
                        int2 ew[kBatchUnroll];
                        int dq[kBatchUnroll], qq[kBatchUnroll], cd[kBatchUnroll];
                        bool ok[kBatchUnroll];
#pragma unroll
                        for (int u = 0; u < kBatchUnroll; ++u) {
                            ok[u] = (unsigned)eis[u] < len;
                            ew[u] = ok[u] ? __ldg(eadj + eis[u]) : make_int2(0, 0);
                        }
#pragma unroll
                        for (int u = 0; u < kBatchUnroll; ++u) {
                            dq[u] = __shfl_sync(kFull, du, js[u]);
                            qq[u] = __shfl_sync(kFull, qp, js[u]);
                        }
#pragma unroll
                        for (int u = 0; u < kBatchUnroll; ++u)
                            cd[u] = ok[u] ? ldcg(dw + (size_t)(unsigned)ew[u].x * Qu + qq[u]) : INT_MIN;
#pragma unroll
                        for (int u = 0; u < kBatchUnroll; ++u) {
                            const int nd = dq[u] + ew[u].y;
                            if (nd < cd[u]) {
                                atomicMin(dw + (size_t)(unsigned)ew[u].x * Qu + qq[u], nd);
                                atomicOr(mrow + ((size_t)(unsigned)ew[u].x << p.logW), 1u << qq[u]);
                                if (low && nd < qlow[(w << 5) + qq[u]]) atomicMin(&qlow[(w << 5) + qq[u]], nd);
                            }
                        }
                    });
                    if (lane == 0) relax += (long long)cnt * len;
                    steps += len;
                }
                e0 = seg_end;
                o += 32;
            }
        }
        if (low) {  // the block's smallest new distances join the next round's qmin
            __syncthreads();
            int* q = p.qmin + ((cur + 1) % 3) * Qu;
            for (unsigned i = threadIdx.x; i < Qu; i += blockDim.x) {
                const int x = qlow[i];
                if (x < ldcg(q + i)) atomicMin(q + i, x);
                qlow[i] = INT_MAX;
            }
        }
        }
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        phase_mark(ctl->phase_ns, tph, 2);
        if (gtid == 0) trace_mid(p.trace, iters - 1);
        ++cur;
        // end of an epoch: the next round's improvements wait in the masks
        if (p.epoch_rounds > 0 && iters >= p.epoch_rounds) break;
    }
    // relax is counted by lane 0 of each warp
    if (lane == 0) {
        atomicAdd((unsigned long long*)&p.counters[0], (unsigned long long)relax);
        atomicAdd((unsigned long long*)&p.counters[1], (unsigned long long)steps);
    }
    if (gtid == 0) {
        ctl->iterations = iters;
        trace_round(p.trace, iters, 0, -1);
    }
}

// Copy dist[V][Q] (first nq queries) into the caller's layout.
__global__ void batch_transpose(const int* __restrict__ dist, int V, int Q, int nq, int* __restrict__ out,
                                int query_major) {
    const size_t total = (size_t)V * (size_t)nq;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        if (query_major) {
            const size_t qi = i / (size_t)V, v = i % (size_t)V;  // coalesced writes
            out[i] = dist[v * Q + qi];
        } else {
            const size_t v = i / (size_t)nq, qi = i % (size_t)nq;
            out[i] = dist[v * Q + qi];
        }
    }
}

// [V][Q] state -> query-major [nq][V] output through a 32 x 32 shared-memory tile: the
// reads cover one 128-byte line of 32 queries per vertex, the writes 32 consecutive
// vertices per query, both coalesced.  (Element-wise, consecutive threads would read with
// a stride of one vertex row.)  Block 32 x 8; grid (V / 32, nq / 32), rounded up.
template <typename S, typename D>
__global__ void __launch_bounds__(256) batch_transpose_qmajor(const S* __restrict__ src, int V, int Q, int nq,
                                                             D* __restrict__ out) {
    __shared__ D tile[32][33];
    const int v0 = (int)blockIdx.x * 32, q0 = (int)blockIdx.y * 32;
    for (int k = (int)threadIdx.y; k < 32; k += 8) {
        const int v = v0 + k, q = q0 + (int)threadIdx.x;
        if (v < V && q < nq) tile[k][threadIdx.x] = (D)src[(size_t)v * (size_t)Q + (size_t)q];
    }
    __syncthreads();
    for (int k = (int)threadIdx.y; k < 32; k += 8) {
        const int q = q0 + k, v = v0 + (int)threadIdx.x;
        if (q < nq && v < V) out[(size_t)q * (size_t)V + (size_t)v] = tile[threadIdx.x][k];
    }
}

// A host output buffer the kernels can write directly: page-locked host memory has a
// device address (over NVLink-C2C on Grace machines), so the results skip the device
// staging copy and the separate device-to-host copy.  nullptr for pageable memory.
static void* mapped_host(void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();  // clear the error state of the query
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

template <typename S, typename D>
static void launch_transpose_qmajor(const S* src, int V, int Q, int nq, D* out, cudaStream_t st) {
    if (V <= 0 || nq <= 0) return;
    const dim3 grid((unsigned)((V + 31) / 32), (unsigned)((nq + 31) / 32));
    batch_transpose_qmajor<S, D><<<grid, dim3(32, 8), 0, st>>>(src, V, Q, nq, out);
}

// ---------------------------------------------------------------------------------------
// host side

// Blocks of a batched launch: the whole GPU, or the handle's share when several
// batched launches run side by side (the serving loop).
static int grid_blocks(const c2g_graph* g, int per_sm) {
    int b = (int)((float)(per_sm * g->num_sms) * g->grid_scale);
    return b < 1 ? 1 : b;
}

// The kernel for queries in the first nq slots: pulls take as many words at a time as hold queries.
static const void* sssp_batch_kernel(int nq) {
    return nq <= 32 ? (const void*)sssp_batch_persistent<1>
         : nq <= 64 ? (const void*)sssp_batch_persistent<2>
                    : (const void*)sssp_batch_persistent<4>;
}

struct BatchWork {
    int* dist = nullptr;
    unsigned* mask = nullptr;
    int2* q[2] = {nullptr, nullptr};
    unsigned* qmask[2] = {nullptr, nullptr};
    int* mark[2] = {nullptr, nullptr};
    TraversalCtl* ctl = nullptr;
    long long* counters = nullptr;
    int* src = nullptr;
    int* seed_off = nullptr;
    int* seed_v = nullptr;
    int* seed_w = nullptr;
    int* stage = nullptr;  // caller-layout copy for host output
    RoundTrace* trace = nullptr;
    unsigned* amask[2] = {nullptr, nullptr};  // pull rounds' lookups of the frontier's lanes
    int* qmin = nullptr;                      // pull rounds: smallest distance of each query's frontier, 3 slots
    size_t seed_cap = 0;
    int Q = 0;
    int V = 0;
};

static void batch_free_work(BatchWork* w) {
    if (!w) return;
    void* ptrs[] = {w->dist, w->mask, w->q[0], w->q[1], w->qmask[0], w->qmask[1], w->mark[0], w->mark[1],
                    w->ctl, w->counters, w->src, w->seed_off, w->seed_v, w->seed_w, w->stage, w->trace,
                    w->amask[0], w->amask[1], w->qmin};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete w;
}

void batch_free(c2g_graph* g) {
    BatchWork* w = reinterpret_cast<BatchWork*>(g->batch);
    if (w && g->last_trace == w->trace) g->last_trace = nullptr;
    batch_free_work(w);
    g->batch = nullptr;
}

static int batch_alloc(c2g_graph* g, int Q, size_t n_seeds) {
    BatchWork* w = reinterpret_cast<BatchWork*>(g->batch);
    if (w && w->Q >= Q && w->seed_cap >= n_seeds) return C2G_OK;
    if (w) batch_free(g);
    w = new BatchWork();
    g->batch = w;
    const size_t V = g->V ? (size_t)g->V : 1;
    const size_t W = (size_t)Q / 32;
    const size_t qcap = V * W;
    const size_t mark_cap = (((size_t)g->E * W) >> kBatchTileLog) + 2;
    C2G_CUDA(cudaMalloc(&w->dist, sizeof(int) * V * (size_t)Q));
    C2G_CUDA(cudaMalloc(&w->mask, sizeof(unsigned) * qcap));
    for (int b = 0; b < 2; ++b) {
        C2G_CUDA(cudaMalloc(&w->q[b], sizeof(int2) * qcap));
        C2G_CUDA(cudaMalloc(&w->qmask[b], sizeof(unsigned) * qcap));
        C2G_CUDA(cudaMalloc(&w->mark[b], sizeof(int) * mark_cap));
    }
    C2G_CUDA(cudaMalloc(&w->ctl, sizeof(TraversalCtl)));
    C2G_CUDA(cudaMalloc(&w->counters, sizeof(long long) * 2));
    C2G_CUDA(cudaMalloc(&w->src, sizeof(int) * (size_t)Q));
    C2G_CUDA(cudaMalloc(&w->seed_off, sizeof(int) * ((size_t)Q + 1)));
    w->seed_cap = n_seeds > 0 ? n_seeds : 1;
    C2G_CUDA(cudaMalloc(&w->seed_v, sizeof(int) * w->seed_cap));
    C2G_CUDA(cudaMalloc(&w->seed_w, sizeof(int) * w->seed_cap));
    C2G_CUDA(cudaMalloc(&w->trace, sizeof(RoundTrace) * (kMaxTraceRounds + 1)));
    for (int b = 0; b < 2; ++b) C2G_CUDA(cudaMalloc(&w->amask[b], sizeof(unsigned) * qcap));
    C2G_CUDA(cudaMalloc(&w->qmin, sizeof(int) * 3 * (size_t)Q));
    w->Q = Q;
    w->V = g->V;
    return C2G_OK;
}

// (query, edge) relaxations above which a round pulls: batch_pull_frac * E * Q, times the
// batch's width factor.  A pull's cost is its pass over the V * W (vertex, word) lines, a push's its
// relaxations, and a wide batch amortises the pass: measured (push only / 0.3 / 0.1 / 0.03 of
// E * Q): scale 22, 256 queries 137 / 60.3 / 53.2 / 44.3 ms; 500,003 uniform vertices, 256 queries
// 27.4 / 22.3 / 21.6 / 21.3; scale 19, 64 queries 5.0 / 3.5 / 3.0 / 3.2; 685,230 uniform vertices, 31
// queries 5.1 / 5.2 / - / 5.8.  After a launch's first pull the distances bound the rows
// of the next ones, whose passes get shorter (scale 22, 256 queries: 7.8 ms, then 4.0, 2.9, 2.6), so a
// batch of one or two words goes on pulling down to the wide one's limit: scale 21, 64 queries 9.15 -> 7.95
// ms, 32 6.60 -> 5.91; for 256 a lower limit is no gain (500,003 uniform vertices 25.0, a third of it 26.6).
//
// At the default fraction two kinds of batches expand only.  (1) Small ones, where the warps with the longest rows
// outlast the rest of a pull: fewer than kPullMinLines lines, unless the queries together relax so much in a full
// round that the push is the longer one all the same (expand only / pull: 65,536 vertices of scale 16, 250 queries, 239 M
// relaxations 2.21 / 2.29 ms; 100,000 uniform vertices, 130 of degree 15, 195 M 3.26 / 3.60, 250, 375 M 5.58 / 4.74, 250 of degree
// 40, 1.0 G 10.0 / 5.5; 60,000 of degree 60, 70, 252 M 2.51 / 2.70, 250, 900 M 7.35 / 3.92; two words, 60 queries, 210 -
// 225 M: scale 18 1.94 / 1.60, 250,000 uniform 3.81 / 3.23, 30,000 1.59 / 1.39).  (2) One word on a graph without hubs,
// whose rounds never get dense enough (in_hubs; 1M uniform vertices, 12 / 31 queries 5.5 / 7.0, 7.2 / 8.0; 2M 11.4 /
// 14.5, 16.4 / 17.8; 4M 18.4 / 19.1, 24.4 / 26.3).
constexpr size_t kPullMinLines = 1000000;
constexpr unsigned long long kPullMinReach2 = 200000000ull, kPullMinReach4 = 300000000ull;  // of 2 and of more words

// A resident batch goes by the words up to its last running slot, not by its slots (Q here): with all slots' pull
// limits and words 11 queries in 256 slots pulled 8 words of which one was at work (scale 18: 0.92 ms with expansion
// only, 1.46 so).
static void sssp_pull_min(const c2g_graph* g, int Q, int queries, unsigned long long* first, unsigned long long* next) {
    *first = *next = ~0ull;
    const float frac = g->sssp_cfg.batch_pull_frac;
    const unsigned long long reach = (unsigned long long)queries * (unsigned long long)g->E;
    const bool small = frac == kDefaultPullFrac && (size_t)g->V * (size_t)(Q / 32) < kPullMinLines &&
                       (Q <= 32 || reach < (Q <= 64 ? kPullMinReach2 : kPullMinReach4));
    if (!(frac >= 0.f) || small) return;
    const double width = Q <= 32 ? 1.0 : Q <= 64 ? 1.0 / 3.0 : 0.1, all = (double)frac * (double)g->E * (double)Q;
    *first = (unsigned long long)(width * all);
    *next = (unsigned long long)(0.1 * all);
}

// The pull rounds of a batched SSSP launch (p.pull_min: (query, edge) relaxations of the
// frontier above which a round pulls, ~0: never): they need the graph's in-edge rows, and
// seeds that are not below zero (the frontier minima start at 0).  The pull
// lookups start clear; a launch leaves the entries of its last rounds behind.  Qrule: the queries the limits go by;
// queries: those at work, which all together cannot pass the limit when they are few: such a launch keeps no lookup.
static int sssp_pull_setup(c2g_graph* g, BatchWork* w, int Q, int Qrule, int queries, bool seeds, BatchParams& p) {
    p.pull_min = ~0ull;
    unsigned long long pull_min, pull_next;
    sssp_pull_min(g, Qrule, queries, &pull_min, &pull_next);
    if ((unsigned long long)queries * (unsigned long long)g->E <= pull_min) pull_min = ~0ull;
    int rc;
    if (pull_min != ~0ull && (rc = ensure_in_rows(g))) return rc;
    if (pull_min == ~0ull || !g->in_adj || (seeds && g->hw_negative)) return C2G_OK;
    if (Qrule <= 32 && !g->in_hubs && g->sssp_cfg.batch_pull_frac == kDefaultPullFrac) return C2G_OK;
    p.in_row = g->in_row;
    p.in_adj = g->in_adj;
    p.in_seg = g->in_seg;
    p.in_segs = g->in_segs;
    p.in_shift = g->in_shift;
    p.qmin = w->qmin;
    for (int b = 0; b < 2; ++b)
        C2G_CUDA(cudaMemsetAsync(w->amask[b], 0, sizeof(unsigned) * (size_t)g->V * (size_t)(Q / 32), g->stream));
    p.pull_min = pull_min;
    p.pull_next = pull_next;
    const unsigned words = ((unsigned)p.nq + 31u) / 32u;
    p.pull_groups = words <= 2u ? 1u : (words + 3u) / 4u;
    return C2G_OK;
}

static void sssp_batch_params(c2g_graph* g, BatchWork* w, int Q, int logW, BatchParams& p) {
    p.row = g->row;
    p.adj = g->adj_w;
    p.E = (unsigned)g->E;
    p.V = g->V;
    p.logW = logW;
    p.Q = Q;
    p.nq = Q;
    for (unsigned& live : p.live) live = ~0u;
    p.dist = w->dist;
    p.mask = w->mask;
    for (int b = 0; b < 2; ++b) {
        p.q[b] = w->q[b];
        p.qmask[b] = w->qmask[b];
        p.mark[b] = w->mark[b];
    }
    p.ctl = w->ctl;
    p.sources = w->src;
    p.seed_off = nullptr;
    p.seed_v = w->seed_v;
    p.seed_w = w->seed_w;
    p.qcap = (unsigned)((size_t)g->V * (size_t)(Q / 32));
    p.mark_cap = (unsigned)((((size_t)g->E * (size_t)(Q / 32)) >> kBatchTileLog) + 2);
    p.max_iter = g->sssp_cfg.max_iter;
    p.barrier_ns = g->barrier_ns ? g->barrier_ns : 4000000000ull;
    p.counters = w->counters;
    p.tile_big_log = g->sssp_cfg.batch_tile_big_log;
    p.tile_min_log = g->sssp_cfg.batch_tile_min_log;
    p.epoch_rounds = 0;
    p.trace = w->trace;
    g->last_trace = w->trace;
    p.in_row = nullptr;  // set by sssp_pull_setup when the launch may pull
    p.in_adj = nullptr;
    p.in_seg = nullptr;
    p.in_segs = 0u;
    p.in_shift = 0;
    p.pull_groups = 0u;
    p.qmin = nullptr;
    p.pull_min = ~0ull;
    p.amask[0] = w->amask[0];
    p.amask[1] = w->amask[1];
}

static int sssp_batch_results(c2g_graph* g, BatchWork* w, int Q, int32_t nq, int32_t* out, int out_on_device,
                              int query_major, float* ms, long long* counters, TraversalCtl* ctl_out) {
    // Results in the caller's layout (pinned host memory is written directly).
    int* dst = out;
    int* direct = out_on_device ? nullptr : static_cast<int*>(mapped_host(out));
    if (direct) {
        dst = direct;
    } else if (!out_on_device) {
        if (!w->stage) C2G_CUDA(cudaMalloc(&w->stage, sizeof(int) * (size_t)g->V * (size_t)Q));
        dst = w->stage;
    }
    if (query_major)
        launch_transpose_qmajor<int, int>(w->dist, g->V, Q, nq, dst, g->stream);
    else
        batch_transpose<<<g->num_sms * 8, 256, 0, g->stream>>>(w->dist, g->V, Q, nq, dst, query_major);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && !out_on_device && !direct)
        e = cudaMemcpyAsync(out, dst, sizeof(int) * (size_t)g->V * (size_t)nq, cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctl_out, w->ctl, sizeof(TraversalCtl), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(counters, w->counters, sizeof(long long) * 2, cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    C2G_CUDA(e);
    C2G_CUDA(cudaEventElapsedTime(ms, g->ev0, g->ev1));
    return C2G_OK;
}

int sssp_batch_launch(c2g_graph* g, int32_t nq, const int32_t* sources, const std::vector<int32_t>* seed_off,
                      const std::vector<int32_t>* seed_v, const std::vector<int32_t>* seed_w, int32_t* out,
                      int out_on_device, int query_major, float* ms, long long* counters, TraversalCtl* ctl_out) {
    if (!g->adj_w) return fail(C2G_ERR_UNSUPPORTED, "graph has no int32 weights (wlist)");
    int Q = 32, logW = 0;
    while (Q < nq) {
        Q <<= 1;
        ++logW;
    }
    if ((size_t)g->V * (size_t)(Q / 32) >= (size_t(1) << 31) || (size_t)g->E * (size_t)(Q / 32) >= (size_t(1) << 32))
        return fail(C2G_ERR_RANGE, "batch of %d queries too large for this graph", nq);
    int rc;
    const size_t ns = seed_v ? seed_v->size() : 0;
    if ((rc = batch_alloc(g, Q, ns))) return rc;
    BatchWork* w = reinterpret_cast<BatchWork*>(g->batch);
    int coop = 0, per_sm = 0;
    C2G_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g->device));
    if (!coop) return fail(C2G_ERR_UNSUPPORTED, "device lacks cooperative launch");
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sssp_batch_kernel(nq), kSsspBatchThreads, 0));
    if (per_sm < 1) return fail(C2G_ERR_CUDA, "batch kernel cannot be resident");

    C2G_CUDA(cudaMemcpyAsync(w->src, sources, sizeof(int) * (size_t)nq, cudaMemcpyHostToDevice, g->stream));
    if (seed_off) {
        C2G_CUDA(cudaMemcpyAsync(w->seed_off, seed_off->data(), sizeof(int) * seed_off->size(),
                                 cudaMemcpyHostToDevice, g->stream));
        if (ns) {
            C2G_CUDA(cudaMemcpyAsync(w->seed_v, seed_v->data(), sizeof(int) * ns, cudaMemcpyHostToDevice, g->stream));
            C2G_CUDA(cudaMemcpyAsync(w->seed_w, seed_w->data(), sizeof(int) * ns, cudaMemcpyHostToDevice, g->stream));
        }
    }
    BatchParams p;
    sssp_batch_params(g, w, Q, logW, p);
    p.nq = nq;
    if ((rc = sssp_pull_setup(g, w, Q, Q, nq, seed_off != nullptr, p))) return rc;
    p.seed_off = seed_off ? w->seed_off : nullptr;
    C2G_CUDA(cudaMemsetAsync(w->ctl, 0, sizeof(TraversalCtl), g->stream));
    C2G_CUDA(cudaMemsetAsync(w->counters, 0, sizeof(long long) * 2, g->stream));
    void* args[] = {&p};
    C2G_CUDA(cudaEventRecord(g->ev0, g->stream));
    const int blocks = grid_blocks(g, per_sm);
    C2G_CUDA(cudaLaunchCooperativeKernel(sssp_batch_kernel(nq), dim3(blocks), dim3(kSsspBatchThreads),
                                         args, 0, g->stream));
    C2G_CUDA(cudaEventRecord(g->ev1, g->stream));
    return sssp_batch_results(g, w, Q, nq, out, out_on_device, query_major, ms, counters, ctl_out);
}

// Resident batch (c2g_session): the workspace of Q query slots with every mask clear, and
// one epoch of at most `rounds` rounds from the state the previous epoch left.
int sssp_batch_reserve(c2g_graph* g, int Q, int** dist, unsigned** mask) {
    if (!g->adj_w) return fail(C2G_ERR_UNSUPPORTED, "graph has no int32 weights (wlist)");
    if ((size_t)g->V * (size_t)(Q / 32) >= (size_t(1) << 31) || (size_t)g->E * (size_t)(Q / 32) >= (size_t(1) << 32))
        return fail(C2G_ERR_RANGE, "%d slots too many for this graph", Q);
    int rc;
    if ((rc = batch_alloc(g, Q, 0))) return rc;
    BatchWork* w = reinterpret_cast<BatchWork*>(g->batch);
    C2G_CUDA(cudaMemsetAsync(w->mask, 0, sizeof(unsigned) * (size_t)g->V * (size_t)(Q / 32), g->stream));
    C2G_CUDA(cudaStreamSynchronize(g->stream));
    *dist = w->dist;
    *mask = w->mask;
    return C2G_OK;
}

int sssp_batch_epoch(c2g_graph* g, int Q, int used, int running, const unsigned* live, int rounds, float* ms,
                     long long* counters, TraversalCtl* ctl_out) {
    BatchWork* w = reinterpret_cast<BatchWork*>(g->batch);
    if (!w || w->Q < Q) return fail(C2G_ERR_ARG, "resident SSSP batch has no workspace");
    int logW = 0;
    while ((32 << logW) < Q) ++logW;
    int per_sm = 0;
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sssp_batch_kernel(used), kSsspBatchThreads, 0));
    if (per_sm < 1) return fail(C2G_ERR_CUDA, "batch kernel cannot be resident");
    BatchParams p;
    sssp_batch_params(g, w, Q, logW, p);
    int rc;
    p.nq = used;
    std::memcpy(p.live, live, sizeof(p.live));
    if ((rc = sssp_pull_setup(g, w, Q, std::max(32, (used + 31) / 32 * 32), running, false, p))) return rc;
    p.epoch_rounds = rounds < 1 ? 1 : rounds;
    C2G_CUDA(cudaMemsetAsync(w->ctl, 0, sizeof(TraversalCtl), g->stream));
    C2G_CUDA(cudaMemsetAsync(w->counters, 0, sizeof(long long) * 2, g->stream));
    void* args[] = {&p};
    C2G_CUDA(cudaEventRecord(g->ev0, g->stream));
    C2G_CUDA(cudaLaunchCooperativeKernel(sssp_batch_kernel(used), dim3(grid_blocks(g, per_sm)),
                                         dim3(kSsspBatchThreads), args, 0, g->stream));
    C2G_CUDA(cudaEventRecord(g->ev1, g->stream));
    C2G_CUDA(cudaMemcpyAsync(ctl_out, w->ctl, sizeof(TraversalCtl), cudaMemcpyDeviceToHost, g->stream));
    C2G_CUDA(cudaMemcpyAsync(counters, w->counters, sizeof(long long) * 2, cudaMemcpyDeviceToHost, g->stream));
    C2G_CUDA(cudaStreamSynchronize(g->stream));
    C2G_CUDA(cudaEventElapsedTime(ms, g->ev0, g->ev1));
    return C2G_OK;
}

}  // namespace c2g

// =======================================================================================
// Batched forward push (PPR) with per-query bitmask frontiers.
//
// Same BSP semantics per query as c2g_ppr (src/ppr/purn/Main.cu:149-428): pop r, push
// (1-alpha)*r*w into msg, then res += msg; if res > rmax: pr += alpha*res and activate.
// State is vertex-major [V][Q]: pr float; res, msg and rq (the residual being pushed,
// times 1-alpha) FP64.  A push round marks the target's (vertex, word) touched mask with
// red.or; phase B sweeps the touched masks, applies the messages and activates, building
// the frontier entries (vertex, word) with the activated lanes as their mask.  A round
// with many pushes runs as a pull over the reverse CSR instead (pbatch_pull); both shapes
// produce the same rounds.
namespace c2g {

struct PprBatchParams {
    const int* row;
    const int2* adj;  // (target, float weight bits)
    unsigned E;
    int V;
    int logW, Q, nq;
    float* pr;        // [V][Q]
    double* res;      // [V][Q] FP64 residuals (see ppr.cu: threshold decisions)
    double* msg;      // [V][Q], zero between launches (pull rounds: parts of tile-straddling targets)
    double* rq[2];    // [V][Q] (1-alpha) * residual being pushed, by frontier buffer
    float2* rqf[2];   // the same as a float pair hi + lo (pull rounds)
    unsigned* amask[2];  // [V][W] lanes activated with out-edges, by frontier buffer (pull lookup)
    unsigned* tmask;  // [V][W] touched lanes this round, zero between rounds
    unsigned* slist;  // pull rounds: the (vertex, word)s a pull left in tmask (tile-straddling targets)
    unsigned slist_cap;
    unsigned* dmask;  // [V][W] lanes activated without out-edges (popped next round), zero between launches
    int2* q[2];       // frontier entries (v*W + w, edge base)
    unsigned* qmask[2];
    int* mark[2];
    int2* dangle;     // (v*W + w, lanes) activated without out-edges, popped next round
    TraversalCtl* ctl;
    const int* sources;
    const int* seed_off;  // seeded mode: per-query record offsets
    const int* seed_v;
    const float* seed_w;
    float alpha, rmax, r0, pr0;
    int seeded;
    int max_iter;
    unsigned qcap, mark_cap;
    unsigned long long barrier_ns;
    long long* counters;  // [2] pushes (query, edge), edge-word steps
    // pull rounds: reverse CSR (source, weight bits); a round pulls when its pushes exceed
    // pull_min
    const int2* adj_r;
    const unsigned* r_bits;   // per chunk of 32 in-edges: which start a row,
    const int* r_prefix;      // how many rows start in earlier chunks,
    const int* r_rows;        // and the rows in order
    int pull_log;             // log2 of the chunks per pull item
    unsigned pull_groups;     // groups of WP query words with queries
    unsigned long long pull_min;
    int epoch_rounds;  // > 0: an epoch of a resident batch (state at rest in the arrays; at most this many rounds)
    int cur0;          // round index the epoch starts at (its parity picks the frontier buffers)
    RoundTrace* trace;  // [kMaxTraceRounds + 1] per-round trace
};

__device__ __forceinline__ FrontierOut pbatch_out(const PprBatchParams& p, int buf, int slot) {
    FrontierOut o;
    o.q = p.q[buf];
    o.val = reinterpret_cast<float*>(p.qmask[buf]);  // mask bits travel in the value slot
    o.mark = p.mark[buf];
    o.ctr = &p.ctl->qctr[slot];
    o.cap = p.qcap;
    o.mark_cap = p.mark_cap;
    o.log_tile = kBatchTileLog;
    o.flags = &p.ctl->flags;
    return o;
}

// Launch shape of the batched PPR: 2 blocks of 448 threads per SM (72 registers).  Measured with the
// pull rounds' chunk streams, 256 queries at scale 21 / 40 at scale 16: 448 threads 368 / 10.0 ms, 512
// (64 registers, more spills) 383 / 10.8, 384 390 / 9.7; 3 x 384 and 4 x 256 lost before that.
constexpr int kPprBatchThreads = 448;
constexpr int kPprBatchBlocksPerSm = 2;
constexpr int kPprBatchUnroll = 3;  // push items in flight per lane
constexpr unsigned long long kPullsEnd = 1ull << 63;  // beside a round's push count: a residual too large for pulls
constexpr unsigned long long kPullMaxQBits = (unsigned long long)((kPullMaxQ >> 23) - 127 + 1023) << 52;  // as a double

// Apply of one (vertex, word) to the lanes that received messages: res += m; a lane whose
// residual exceeds rmax adds alpha * res to pr and activates.  An activated lane with
// out-edges stores (1-alpha) * res as the residual it pushes next round (in rq[ob]) and
// zeroes res; one without out-edges keeps res until the next round pops it.  The word's
// activated lanes go to the next frontier (and to amask[ob], the pull rounds' lookup),
// or to the dangling list.  force = true: the seeded first hop (activate every touched
// lane, no messages).  psum (lane 0) accumulates the next round's pushes.  WP < 4: a residual too large for the
// pulls' float pairs makes the next round and those after it push, as in ppr.cu.  Batches of up to 64 queries need
// that, which pull from few pushes on (ppr_pull_threshold); in the kernel of wider ones, which pull above 8 E
// pushes as they always have, the test took 1% of a batch (256 queries at scale 21: 372 -> 377 ms).
template <int WP>
__device__ __forceinline__ void pbatch_apply_word(const PprBatchParams& p, bool force, int ob, int vw, int dg,
                                                  size_t off, bool mine, double r, double m, float pv,
                                                  unsigned long long rmax_bits, WarpStage& fst, const FrontierOut& out,
                                                  unsigned* dctr, unsigned long long& psum, int lane) {
    bool act = false;
    if (mine) {
        double rr = r;
        if (!force) rr += m;
        // rr and rmax are non-negative: compare their bit patterns
        if (force || c2g_dbits(rr) > rmax_bits) {
            if (!force) p.pr[off] = pv + (float)((double)p.alpha * rr);
            act = true;
            if (dg > 0) {
                const double q = (1.0 - (double)p.alpha) * rr;  // (1-alpha)*r_u (src/ppr/purn/Main.cu:288)
                p.rq[ob][off] = q;
                if (c2g_split_ok(q) && (WP == 4 || c2g_dbits(q) < kPullMaxQBits)) {  // float pair for pull rounds (fp64_mul.h)
                    const c2g_pair hl = c2g_split_pair(q);
                    p.rqf[ob][off] = make_float2(c2g_bitsf(hl.hi), c2g_bitsf(hl.lo));
                } else {
                    const float hi = __double2float_rz(q);
                    p.rqf[ob][off] = make_float2(hi, __double2float_rz(q - (double)hi));
                    // too large for the pairs' sums: the next round and those after it push (ppr.cu)
                    if (WP < 4 && c2g_dbits(q) >= kPullMaxQBits) atomicOr(&p.ctl->pcount[dctr - p.ctl->dctr], kPullsEnd);
                }
                p.res[off] = 0.0;
            } else {
                p.res[off] = rr;  // popped (zeroed) at the top of the next round
            }
        } else {
            p.res[off] = rr;
        }
    }
    const unsigned bits = __ballot_sync(kFull, act);
    if (bits && lane == 0) {
        if (dg == 0) {
            const unsigned slot = atomicAdd(dctr, 1u);
            if (slot < p.qcap)
                p.dangle[slot] = make_int2(vw, (int)bits);
            else
                atomicOr(&p.ctl->flags, C2G_FLAG_QUEUE_OVERFLOW);
            p.dmask[vw] = bits;  // the same lanes at rest, for an epoch boundary
        } else {
            p.amask[ob][vw] = bits;
            psum += (unsigned long long)__popc(bits) * (unsigned long long)dg;
        }
    }
    stage_push(fst, out, lane == 0 && bits != 0u && dg > 0, vw, dg, __int_as_float((int)bits));
}

// Apply sweep: every (vertex, word) whose touched mask is non-zero applies its messages
// lane by lane (lane = query) and activates; the mask is cleared.  Pushes mark targets with
// red.or, so the push never waits on an atomic's return; the sweep reads V * W mask words
// per round.  After a pull round only the targets whose in-edges cross a tile boundary
// are left, and the sweep visits just those, from the list the pull wrote (list != null:
// nlist word indices; 842 vs 875 ms per 256-query batch at scale 22 against sweeping all
// V * W words).  A warp takes 32 words at a time (their degrees loaded lane-parallel) and
// applies up to kApplyGroup touched words at once: all their residual, message and pr
// loads are issued before any of them is used, so the words' memory latencies overlap
// instead of adding up.  (Loading 2 or 4 blocks of 32 mask words before applying any
// measured slower: 852 and 870 ms.)
constexpr int kApplyGroup = 3;  // 4 spills at 64 registers

template <int WP>
__device__ __forceinline__ unsigned pbatch_sweep(const PprBatchParams& p, bool force, int ob, const unsigned* list,
                                                 unsigned nlist, WarpStage& fst, const FrontierOut& out,
                                                 unsigned* dctr, unsigned long long& psum, unsigned gwarp,
                                                 unsigned nwarps, int lane) {
    const unsigned nm = list ? nlist : (unsigned)p.V << p.logW;
    const unsigned long long rmax_bits = c2g_dbits((double)p.rmax);
    unsigned cnt = 0;
    // words a warp takes at a time: every listed word costs an apply, so a list is spread over all warps
    // (50,000 words on 4,256 warps, 40 queries at scale 16: 65 us a round at 32 each, 23 so; a mask word
    // of a whole sweep is mostly empty)
    const unsigned rounds = (nm + nwarps * 32u - 1u) / (nwarps * 32u);
    const unsigned take = list ? (nm + nwarps * rounds - 1u) / max(1u, nwarps * rounds) : 32u;
    for (unsigned b = gwarp * take; b < nm; b += nwarps * take) {
        const unsigned pos = b + (unsigned)lane;
        const bool in = (unsigned)lane < take && pos < nm;
        const unsigned i = in ? (list ? ldcg(list + pos) : pos) : 0u;  // this lane's (vertex, word)
        const unsigned tm = in ? ldcg(p.tmask + i) : 0u;
        int dg = 0;
        if (tm) {
            p.tmask[i] = 0u;
            const int v = (int)(i >> p.logW);
            dg = __ldg(p.row + v + 1) - __ldg(p.row + v);
        }
        unsigned nz = __ballot_sync(kFull, tm != 0u);
        cnt += (unsigned)__popc(tm);  // touched (vertex, query) lanes seen by this lane
        while (nz) {
            int ks[kApplyGroup];
#pragma unroll
            for (int u = 0; u < kApplyGroup; ++u) {
                ks[u] = nz ? __ffs(nz) - 1 : -1;
                nz &= nz - 1u;
            }
            // element (v, w*32 + lane) of a [V][Q] array sits at (v*W + w)*32 + lane
            double r[kApplyGroup], m[kApplyGroup];
            float pv[kApplyGroup];
#pragma unroll
            for (int u = 0; u < kApplyGroup; ++u) {
                const int k = ks[u] < 0 ? 0 : ks[u];
                const unsigned ln = ks[u] < 0 ? 0u : (unsigned)__shfl_sync(kFull, (int)tm, k);
                const unsigned vw = (unsigned)__shfl_sync(kFull, (int)i, k);
                const size_t off = ((size_t)vw << 5) + lane;
                const bool mine = (ln >> lane) & 1u;
                r[u] = mine ? ldcg(p.res + off) : 0.0;
                m[u] = (mine && !force) ? ldcg(p.msg + off) : 0.0;
                pv[u] = (mine && !force) ? ldcg(p.pr + off) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kApplyGroup; ++u) {
                if (ks[u] < 0) break;  // warp-uniform
                const unsigned ln = (unsigned)__shfl_sync(kFull, (int)tm, ks[u]);
                const int dgu = __shfl_sync(kFull, dg, ks[u]);
                const int vw = __shfl_sync(kFull, (int)i, ks[u]);
                const size_t off = ((size_t)(unsigned)vw << 5) + lane;
                const bool mine = (ln >> lane) & 1u;
                if (mine && !force) p.msg[off] = 0.0;
                pbatch_apply_word<WP>(p, force, ob, vw, dgu, off, mine, r[u], m[u], pv[u], rmax_bits, fst, out, dctr,
                                  psum, lane);
            }
        }
    }
    stage_flush(fst, out);
    return cnt;
}

// ---------------------------------------------------------------------------------------
// Pull round.  In the dense middle of a batch most (vertex, query) pairs are active, and a
// push does one FP64 read-modify-write per (edge, query) on a message array far larger
// than L2.  A pull round instead walks the reverse CSR: for each target v and query word,
// the warp reads v's in-edges (u, w(u,v)), looks up u's active lanes (amask) and gathers
// the pushed residuals of those lanes (one coalesced 256-byte row segment per edge and
// word), summing the messages rq * w in registers.  The sums are float pairs hi + lo
// (about 47 bits of relative precision): the product is hi*w + lo*w with its rounding
// error recovered by an FMA, and each add is an error-free two-sum whose error joins lo.
// Relative precision matters here, not absolute: a message sum decides res > rmax at the
// scale of rmax, far below the largest sums.
//
// In-edges are cut into chunks of 32 and items of 2^pull_log chunks; warps take (item, group of
// 4 query words) from the round's queue.  Within a warp the chunks form one stream: while a
// chunk is summed, the next one's activity masks and the one after's in-edges are copied to
// shared memory (cp.async: no registers held), across rows and items alike; the row
// boundaries inside a chunk come from one word of start bits, not from the row pointer.
// (Row by row, each row cost a chain of three dependent loads before its first gather, and
// narrow batches left most of an item's 4 words empty: 40 queries at scale 16 took 28.0 ms a
// batch, now 8.4; 256 at scale 21 395, now 368.)  What bounds a dense round of a wide batch is
// the gathers' bytes, 8 per push, at about 6 TB/s out of L2, and about 60 instructions per
// (in-edge, item).  A target whose in-edges lie in one item is applied by the warp that summed
// them; only targets whose in-edges cross an item boundary add their parts to msg (FP64
// atomics) for the apply sweep that follows, as after a push.
constexpr int kPullInFlight = 8;  // (in-edge, query word) rows gathered before they are summed

struct PPullSmem {  // one warp's
    uint4 mk[2][32];  // sources' active lanes of a chunk
    int2 ed[3][32];   // in-edges (source, weight bits) of a chunk
};

// Owner v's message sums of the item's words are complete (hi + lo per lane).  An owner
// whose in-edges lie in this item has them all: it is applied here, by the pulling warp
// (the pullers read the other round parity's rq pairs and activity masks, so this apply
// does not disturb them).  An owner whose in-edges cross an item boundary adds its part to
// msg in FP64 (atomics) and marks tmask; the apply after the barrier finishes it.  The
// first part to mark a (vertex, word) appends it to slist (counter sctr), so that apply
// visits only the listed words instead of sweeping all V * W.  dg: v's out-degree.
template <int WP>
__device__ __forceinline__ unsigned pbatch_pull_owner(const PprBatchParams& p, int v, int dg, unsigned w0, bool whole,
                                                      const float (&sh)[WP], const float (&sl)[WP],
                                                      int ob, unsigned long long rmax_bits, WarpStage& fst,
                                                      const FrontierOut& out, unsigned* dctr, unsigned* sctr,
                                                      unsigned long long& psum, int lane) {
    unsigned cnt = 0;
    if (!whole) {
#pragma unroll
        for (int j = 0; j < WP; ++j) {
            const bool nz = sh[j] != 0.f;
            const unsigned bits = __ballot_sync(kFull, nz);
            if (bits) {
                const size_t vw = ((size_t)(unsigned)v << p.logW) + w0 + j;
                if (nz)
                    atomicAdd(p.msg + (vw << 5) + lane, c2g_float_bits_to_double(__float_as_uint(sh[j])) +
                                                            c2g_float_bits_to_double(__float_as_uint(sl[j])));
                if (lane == 0 && atomicOr(p.tmask + vw, bits) == 0u) {
                    const unsigned k = atomicAdd(sctr, 1u);
                    if (k < p.slist_cap) p.slist[k] = (unsigned)vw;
                }
            }
        }
        return 0;
    }
    double r[WP];
    float pv[WP];
#pragma unroll
    for (int j = 0; j < WP; ++j) {
        const size_t off = (size_t)v * (size_t)p.Q + ((w0 + j) << 5) + lane;
        const bool nz = sh[j] != 0.f;
        r[j] = nz ? ldcg(p.res + off) : 0.0;
        pv[j] = nz ? ldcg(p.pr + off) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < WP; ++j) {
        const bool nz = sh[j] != 0.f;
        if (!__any_sync(kFull, nz)) continue;
        cnt += nz ? 1u : 0u;
        const size_t off = (size_t)v * (size_t)p.Q + ((w0 + j) << 5) + lane;
        const double m = c2g_float_bits_to_double(__float_as_uint(sh[j])) +
                         c2g_float_bits_to_double(__float_as_uint(sl[j]));
        pbatch_apply_word<WP>(p, false, ob, (int)(((unsigned)v << p.logW) + w0 + j), dg, off, nz, r[j], m, pv[j],
                              rmax_bits, fst, out, dctr, psum, lane);
    }
    return cnt;
}

// Two queries' sums s = sh + sl take the messages (hi + lo) * w: the message is pm + pe, then a two-sum of
// sh + pm.  npm = -pm exactly (round-to-nearest is symmetric), so every line rounds as the scalar form
//   pm = hi*w, pe = fma(lo, w, fma(hi, w, -pm)), s = sh + pm,
//   bv = s - sh, av = s - bv, te = (sh - av) + (pm - bv),
//   sl += te + pe, sh = s
// does: pm - bv = -(npm + bv).
__device__ __forceinline__ void pull_pair_add(f32x2 hi, f32x2 lo, f32x2 w, f32x2 nw, f32x2& sh, f32x2& sl) {
    const f32x2 npm = f2_mul(hi, nw);
    const f32x2 pe = f2_fma(lo, w, f2_fma(hi, w, npm));
    const f32x2 s = f2_sub(sh, npm);
    const f32x2 bv = f2_sub(s, sh);
    const f32x2 av = f2_sub(s, bv);
    const f32x2 te = f2_sub(f2_sub(sh, av), f2_add(npm, bv));
    sl = f2_add(sl, f2_add(te, pe));
    sh = s;
}

// The sums of the warp's 32 / LG groups of lanes, two queries per lane, to one query per lane.
template <int LG>
__device__ __forceinline__ void pull_pair_reduce(f32x2 h, f32x2 l, int lane, float& sh, float& sl) {
    float hx, hy, lx, ly;
    f2_unpack(h, hx, hy);
    f2_unpack(l, lx, ly);
#pragma unroll
    for (int o = LG; o < 32; o <<= 1) {
        const f32x2 a = f2_pack(hx, hy);
        const f32x2 b = f2_pack(__shfl_xor_sync(kFull, hx, o), __shfl_xor_sync(kFull, hy, o));
        const f32x2 ol = f2_pack(__shfl_xor_sync(kFull, lx, o), __shfl_xor_sync(kFull, ly, o));
        const f32x2 s = f2_add(a, b), bv = f2_sub(s, a);
        const f32x2 te = f2_add(f2_sub(a, f2_sub(s, bv)), f2_sub(b, bv));
        f2_unpack(s, hx, hy);
        f2_unpack(f2_add(f2_add(f2_pack(lx, ly), ol), te), lx, ly);
    }
    const int src = lane >> 1;
    const float h0 = __shfl_sync(kFull, hx, src), h1 = __shfl_sync(kFull, hy, src);
    const float l0 = __shfl_sync(kFull, lx, src), l1 = __shfl_sync(kFull, ly, src);
    const bool has = lane < 2 * LG;
    sh = has ? (lane & 1 ? h1 : h0) : 0.f;
    sl = has ? (lane & 1 ? l1 : l0) : 0.f;
}

// Position in a warp's stream of chunks.
struct PPullPos {
    unsigned c;   // chunk; ~0: beyond the last item
    unsigned wf;  // first query word of the item's group | kPullFirst | kPullLast (chunk of its item)
};
constexpr unsigned kPullFirst = 1u << 31, kPullLast = 1u << 30;
__device__ __forceinline__ unsigned pull_w0(const PPullPos& q) { return q.wf & ~(kPullFirst | kPullLast); }

// Phase A of a pull round.  LG < 32: a batch of one query word, at most 2 LG queries; LG lanes of two queries each
// take an in-edge, so that a warp takes 32 / LG in-edges at a time and its packed pairs are full (with one query
// per lane a round cost 66 instructions per in-edge for any number of queries: 11 queries at scale 18
// 14.3 -> 11.2 ms a batch, 32 16.6 -> 14.0, 12 at scale 20 42.5 -> 32.0).
template <int WP, int LG>
__device__ __forceinline__ unsigned pbatch_pull(const PprBatchParams& p, int buf, int ob, unsigned* qctr,
                                                PPullSmem& sm, WarpStage& fst, const FrontierOut& out, unsigned* dctr,
                                                unsigned* sctr, unsigned long long& psum, int lane, bool& bad) {
    constexpr int EF = kPullInFlight / WP;  // in-edges in flight
    constexpr int NP = (WP + 1) / 2;        // packed word pairs
    const unsigned nchunks = (p.E + 31u) >> 5;
    const unsigned per_group = (nchunks + (1u << p.pull_log) - 1u) >> p.pull_log;
    const unsigned nitems = per_group * p.pull_groups;
    const unsigned* am = p.amask[buf];
    const float2* rqf = p.rqf[buf];
    const float2* rql = rqf + lane;
    const unsigned lane_bit = 1u << lane;
    const unsigned long long rmax_bits = c2g_dbits((double)p.rmax);
    unsigned cnt = 0;

    unsigned raw = 0;  // lane 0: the next item, taken from the queue ahead of its use
    auto take = [&]() {
        if (lane == 0) raw = atomicAdd(qctr, 1u);
    };
    auto item_start = [&]() {
        unsigned it = (unsigned)__shfl_sync(kFull, (int)raw, 0);
        PPullPos q{~0u, kPullLast};
        if (it < nitems) {
            // from the end of the edge range: items of many short rows cost most (each row is an
            // apply), and in a skewed graph they lie behind the hubs; first, they do not end the
            // round alone (dense rounds, 256 queries: scale 18 2.2 -> 1.6 ms, scale 21 11.3 -> 10.4)
            it = nitems - 1u - it;
            // word group major: all items of one word group, then the next, so the residual
            // rows that L2 holds for the busiest sources are one word group's (1 KB per source,
            // not 2 at 256 queries): 818 vs 843 ms per 256-query batch at scale 22
            q.c = (it % per_group) << p.pull_log;
            q.wf = (it / per_group) * (unsigned)WP | kPullFirst;
            if (p.pull_log == 0 || q.c + 1u == nchunks) q.wf |= kPullLast;
            take();
        }
        return q;
    };
    auto next = [&](const PPullPos& q) {
        if (q.c == ~0u) return q;
        if (q.wf & kPullLast) return item_start();
        PPullPos r{q.c + 1u, q.wf & ~kPullFirst};
        if (((r.c + 1u) & ((1u << p.pull_log) - 1u)) == 0u || r.c + 1u == nchunks) r.wf |= kPullLast;
        return r;
    };
    auto load_edges = [&](const PPullPos& q, int slot) {
        if (q.c == ~0u) return;
        const unsigned e = (q.c << 5) + (unsigned)lane;
        if (e < p.E)
            cp_async8(&sm.ed[slot][lane], p.adj_r + e);
        else
            sm.ed[slot][lane] = make_int2(0, 0);
    };
    auto load_masks = [&](const PPullPos& q, int eslot, int mslot) {
        if (q.c == ~0u) return;
        const int2 e = sm.ed[eslot][lane];
        uint4* to = &sm.mk[mslot][lane];
        if ((unsigned)e.x >= (unsigned)p.V) bad = true;
        if (e.y > 0 && (unsigned)e.x < (unsigned)p.V) {  // positive weights only, as the push
            const unsigned line = ((unsigned)e.x << p.logW) + pull_w0(q);  // the source's first line of the item
            sm.ed[eslot][lane].x = (int)line;
            const unsigned* ms = am + line;
            if (WP == 4)
                cp_async16(to, ms);
            else if (WP == 2)
                cp_async8(to, ms);
            else
                cp_async4(to, ms);
        } else {
            *to = make_uint4(0u, 0u, 0u, 0u);
        }
    };

    take();
    PPullPos q0 = item_start(), q1 = next(q0);
    load_edges(q0, 0);
    load_edges(q1, 1);
    cp_async_commit();
    cp_async_wait_but<0>();
    __syncwarp();
    load_masks(q0, 0, 0);
    cp_async_commit();
    // message sums hi + lo of the words, packed in pairs
    f32x2 sh2[NP], sl2[NP];
    bool whole = false, any = false;  // the row started inside the item; it has a live in-edge
    for (int e0 = 0, m0 = 0; q0.c != ~0u; e0 = e0 == 2 ? 0 : e0 + 1, m0 ^= 1) {
        const int e1 = e0 == 2 ? 0 : e0 + 1, e2 = e1 == 2 ? 0 : e1 + 1;
        const PPullPos q2 = next(q1);
        const unsigned starts = __ldg(p.r_bits + q0.c);
        const unsigned follow = q0.c + 1u < nchunks ? __ldg(p.r_bits + q0.c + 1u) & 1u : 1u;
        const unsigned base = (unsigned)__ldg(p.r_prefix + q0.c) + (starts & 1u) - 1u;
        const unsigned len = min(32u, p.E - (q0.c << 5));
        // the chunk's rows, one per lane: vertex and out-degree
        int rv = 0, rdeg = 0;
        if ((unsigned)lane <= (unsigned)__popc(starts & ~1u)) {
            rv = __ldg(p.r_rows + base + (unsigned)lane);
            rdeg = __ldg(p.row + rv + 1) - __ldg(p.row + rv);
        }
        cp_async_wait_but<0>();  // this chunk's masks, the next one's edges
        __syncwarp();
        load_edges(q2, e2);
        load_masks(q1, e1, m0 ^ 1);
        cp_async_commit();
        unsigned mine;
        {
            const uint4 m = sm.mk[m0][lane];
            mine = WP == 4 ? m.x | m.y | m.z | m.w : WP == 2 ? m.x | m.y : m.x;
        }
        // only in-edges whose source has an active lane in the item's words are visited: the
        // others would add exact zeros
        const unsigned lm = __ballot_sync(kFull, mine != 0u);
        if constexpr (LG < 32) {  // they move to the front, in order: (lanes, line, weight)
            const int2 my = sm.ed[e0][lane];
            const unsigned below = lane_bit - 1u;
            const int at = (lm >> lane) & 1u ? __popc(lm & below) : __popc(lm) + __popc(~lm & below);
            __syncwarp();
            sm.mk[m0][at] = make_uint4(mine, (unsigned)my.x, (unsigned)my.y, 0u);
            __syncwarp();
        }
        if (q0.wf & kPullFirst) {
            whole = false;
            any = false;
#pragma unroll
            for (int j = 0; j < NP; ++j) sh2[j] = sl2[j] = 0ull;
        }
        unsigned pos = 0u;
        for (int i = 0; pos < len; ++i) {
            if ((starts >> pos) & 1u) {
                whole = true;
                any = false;
#pragma unroll
                for (int j = 0; j < NP; ++j) sh2[j] = sl2[j] = 0ull;
            }
            const unsigned after = pos == 31u ? 0u : starts & ~((2u << pos) - 1u);
            const unsigned nxt = after ? (unsigned)__ffs((int)after) - 1u : len;
            unsigned l = lm & (nxt == 32u ? ~0u : (1u << nxt) - 1u) & ~((1u << pos) - 1u);
            any = any || l != 0u;
            if constexpr (LG < 32) {
                constexpr int G = 32 / LG;          // in-edges at a time,
                constexpr int U = G >= 4 ? 2 : 4;   // times U in flight
                const unsigned first = (unsigned)__popc(lm & ((1u << pos) - 1u)), end = first + (unsigned)__popc(l);
                const unsigned q2 = 2u * (unsigned)(lane & (LG - 1));  // this lane's queries q2, q2 + 1
                for (unsigned i0 = first + (unsigned)(lane / LG); i0 - (unsigned)(lane / LG) < end; i0 += G * U) {
                    float4 v[U];
                    float w[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const unsigned i = i0 + (unsigned)(u * G);
                        const uint4 e = i < end ? sm.mk[m0][i] : make_uint4(0u, 0u, 0u, 0u);
                        const unsigned on = (e.x >> q2) & 3u;
                        v[u] = on ? __ldcg(reinterpret_cast<const float4*>(rqf + (size_t)e.y * 32u + q2))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
                        // a query at rest adds exact zeros: its pair here may hold anything (an earlier
                        // query's residual, infinity or NaN), so it is dropped, not weighted with 0
                        if (!(on & 1u)) v[u].x = v[u].y = 0.f;
                        if (!(on & 2u)) v[u].z = v[u].w = 0.f;
                        w[u] = __uint_as_float(e.z);
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        pull_pair_add(f2_pack(v[u].x, v[u].z), f2_pack(v[u].y, v[u].w), f2_pack(w[u], w[u]),
                                      f2_pack(-w[u], -w[u]), sh2[0], sl2[0]);
                }
                l = 0u;
            }
            while (l) {
                // gather the pushed residuals of EF in-edges, then add them
                float2 qb[EF][WP];
                float wk[EF];
#pragma unroll
                for (int h = 0; h < EF; ++h) {
                    const bool have = l != 0u;
                    const int k = __clz((int)__brev(l)) & 31;
                    l &= l - 1u;
                    const int2 ek = sm.ed[e0][k];
                    const uint4 mq = sm.mk[m0][k];
                    wk[h] = __int_as_float(ek.y);
                    const float2* line = rql + (size_t)(unsigned)ek.x * 32u;
                    const unsigned bit = have ? lane_bit : 0u;
#pragma unroll
                    for (int j = 0; j < WP; ++j) {
                        const unsigned mj = j == 0 ? mq.x : j == 1 ? mq.y : j == 2 ? mq.z : mq.w;
                        qb[h][j] = mj & bit ? ldcg(line + 32 * j) : make_float2(0.f, 0.f);
                    }
                }
#pragma unroll
                for (int h = 0; h < EF; ++h) {
                    const f32x2 w2 = f2_pack(wk[h], wk[h]);
                    const f32x2 nw2 = f2_pack(-wk[h], -wk[h]);
#pragma unroll
                    for (int j = 0; j < NP; ++j) {
                        const float2 qa = qb[h][2 * j], qc = 2 * j + 1 < WP ? qb[h][(2 * j + 1) % WP] : make_float2(0.f, 0.f);
                        pull_pair_add(f2_pack(qa.x, qc.x), f2_pack(qa.y, qc.y), w2, nw2, sh2[j], sl2[j]);
                    }
                }
            }
            const bool ends = nxt < len || follow != 0u;
            if (any && (ends || (q0.wf & kPullLast))) {
                float sh[WP], sl[WP];
                if constexpr (LG < 32) pull_pair_reduce<LG>(sh2[0], sl2[0], lane, sh[0], sl[0]);
#pragma unroll
                for (int j = 0; j < NP && LG == 32; ++j) {
                    float a, b, c, d;
                    f2_unpack(sh2[j], a, b);
                    f2_unpack(sl2[j], c, d);
                    sh[2 * j] = a;
                    sl[2 * j] = c;
                    if (2 * j + 1 < WP) {
                        sh[(2 * j + 1) % WP] = b;
                        sl[(2 * j + 1) % WP] = d;
                    }
                }
                cnt += pbatch_pull_owner<WP>(p, __shfl_sync(kFull, rv, i), __shfl_sync(kFull, rdeg, i), pull_w0(q0),
                                             whole && ends, sh, sl, ob, rmax_bits, fst, out, dctr, sctr, psum, lane);
            }
            pos = nxt;
        }
        __syncwarp();
        q0 = q1;
        q1 = q2;
    }
    cp_async_wait_but<0>();
    stage_flush(fst, out);
    return cnt;
}

// Start of an epoch of a resident batch: round `slot`'s frontier from the state at rest,
// the activity masks of buffer b (lanes activated with out-edges, their pushed residuals
// in rq[b] / rqf[b]) and dmask (lanes activated without out-edges), as the apply sweep
// of the previous round would have built it: entries (vertex, word) with their lanes,
// the dangling list, and the round's push count.
__device__ __noinline__ void pbatch_rebuild(const PprBatchParams& p, int b, int slot, WarpStage& fst,
                                               unsigned gwarp, unsigned nwarps, int lane) {
    const unsigned nm = (unsigned)p.V << p.logW;
    const FrontierOut out = pbatch_out(p, b, slot);
    unsigned long long ps = 0;
    for (unsigned base = gwarp * 32u; base < nm; base += nwarps * 32u) {
        const unsigned i = base + (unsigned)lane;
        unsigned a = 0u, d = 0u;
        int deg = 0;
        if (i < nm) {
            a = ldcg(p.amask[b] + i);
            d = ldcg(p.dmask + i);
            if (a) {
                const int v = (int)(i >> p.logW);
                deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
            }
        }
        if (a && deg > 0) ps += (unsigned long long)__popc(a) * (unsigned long long)deg;
        stage_push(fst, out, a != 0u && deg > 0, (int)i, deg, __int_as_float((int)a));
        if (d) {
            const unsigned k = atomicAdd(&p.ctl->dctr[slot], 1u);
            if (k < p.qcap)
                p.dangle[k] = make_int2((int)i, (int)d);
            else
                atomicOr(&p.ctl->flags, C2G_FLAG_QUEUE_OVERFLOW);
        }
    }
    stage_flush(fst, out);
    for (int o = 16; o >= 1; o >>= 1) ps += __shfl_xor_sync(kFull, ps, o);
    if (lane == 0 && ps) atomicAdd(&p.ctl->pcount[slot], ps);
}

// WP: query words of a pull item (1, 2, or 4 of four or more).  Dynamic shared memory: a PPullSmem per warp.
constexpr size_t kPprBatchSmem = sizeof(PPullSmem) * (kPprBatchThreads / 32);

// WP: query words a pull takes at a time (1, 2, or 4 of four or more); LG: lanes of a pulled in-edge (pbatch_pull)
template <int WP, int LG>
__global__ void __launch_bounds__(kPprBatchThreads, kPprBatchBlocksPerSm)
    ppr_batch_persistent(const PprBatchParams p) {
    extern __shared__ uint4 pull_smem[];
    TraversalCtl* ctl = p.ctl;
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(&ctl->bar_count);
    grid_sync_init();
    int* flags = &ctl->flags;
    const int lane = threadIdx.x & 31;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nthreads = gridDim.x * blockDim.x;
    const unsigned gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const int W = 1 << p.logW;
    const unsigned Qu = (unsigned)p.Q;
    __shared__ StageSmem sm;
    const int wib = threadIdx.x >> 5;
    WarpStage fst{sm.v0[wib], sm.d0[wib], sm.x0[wib], 0};
    int* qtab = sm.v1[wib];  // slot -> query position table of the owner being expanded
    PPullSmem& psm = reinterpret_cast<PPullSmem*>(pull_smem)[wib];
    const double one_m_a = 1.0 - (double)p.alpha;
    unsigned long long tph = globaltimer_ns();
    unsigned long long psum = 0;  // next round's pushes counted by this warp (lane 0)

    if (p.epoch_rounds == 0) {
    // Init: pr = res = 0 (msg, tmask, amask and dmask are zero between launches).
    {
        const size_t n4 = ((size_t)p.V * (size_t)p.Q) >> 2;
        float4* a4 = reinterpret_cast<float4*>(p.pr);
        double2* b2 = reinterpret_cast<double2*>(p.res);
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const double2 zd = make_double2(0.0, 0.0);
        for (size_t i = gtid; i < n4; i += nthreads) {
            a4[i] = z;
            b2[2 * i] = zd;
            b2[2 * i + 1] = zd;
        }
    }
    if (!grid_sync(bar, flags, p.barrier_ns)) return;
    // Sources: base mode puts r0 on the source; seeded mode applies the host-side first
    // hop (records + kept out-edges) to pr/res, a warp per query with its lanes over the
    // records and edges (a hub source has thousands).  Either way the touched lanes are
    // marked.
    for (unsigned qi = gwarp; qi < (unsigned)p.nq; qi += nwarps) {
        const int s = p.sources[qi];
        const int w = (int)(qi >> 5);
        const unsigned bit = 1u << (qi & 31);
        if (!p.seeded) {
            if (lane == 0) {
                atomicAdd(p.pr + (size_t)s * p.Q + qi, p.pr0);
                atomicAdd(p.res + (size_t)s * p.Q + qi, (double)p.r0);
                atomicOr(p.tmask + ((size_t)s << p.logW) + w, bit);
            }
        } else {
            if (lane == 0) atomicAdd(p.pr + (size_t)s * p.Q + qi, p.alpha);
            const int rs = __ldg(p.row + s), re = __ldg(p.row + s + 1);
            const int n_rec = p.seed_off[qi + 1] - p.seed_off[qi];
            for (int k = lane; k < n_rec + (re - rs); k += 32) {
                int v;
                float wt;
                if (k < n_rec) {
                    v = p.seed_v[p.seed_off[qi] + k];
                    wt = p.seed_w[p.seed_off[qi] + k];
                } else {
                    const int2 ew = __ldg(p.adj + rs + (k - n_rec));
                    v = ew.x;
                    wt = __int_as_float(ew.y);
                }
                atomicAdd(p.pr + (size_t)v * p.Q + qi, (float)(one_m_a * (double)p.alpha * (double)wt));
                atomicAdd(p.res + (size_t)v * p.Q + qi, one_m_a * (double)wt);
                atomicOr(p.tmask + ((size_t)v << p.logW) + w, bit);
            }
        }
    }
    if (!grid_sync(bar, flags, p.barrier_ns)) return;
    // Round-1 frontier: every touched (vertex, word) activates its touched lanes.
    pbatch_sweep<WP>(p, true, 1, nullptr, 0u, fst, pbatch_out(p, 1, 1), &ctl->dctr[1], psum, gwarp, nwarps, lane);
    if (lane == 0 && psum) atomicAdd(&ctl->pcount[1], psum);
    psum = 0;
    if (!grid_sync(bar, flags, p.barrier_ns)) return;
    } else {
        // An epoch of a resident batch: the state is at rest in the arrays.
        pbatch_rebuild(p, p.cur0 & 1, p.cur0 % 3, fst, gwarp, nwarps, lane);
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
    }
    phase_mark(ctl->phase_ns, tph, 0);

    long long pushes = 0, steps = 0;
    unsigned long long touched = 0;
    int cur = p.epoch_rounds > 0 ? p.cur0 : 1, iters = 0;
    bool bad = false;
    for (;;) {
        const unsigned long long c = ldcg(&ctl->qctr[cur % 3]);
        const unsigned F = (unsigned)(c >> 32), T = (unsigned)c;
        const unsigned D = min(ldcg(&ctl->dctr[cur % 3]), p.qcap);
        const unsigned long long pc = ldcg(&ctl->pcount[cur % 3]);
        const unsigned long long P = pc & ~kPullsEnd;  // this round's (query, edge) pushes
        const bool large = WP < 4 && pc != P;
        if (gtid == 0 && large) atomicOr(&ctl->pcount[(cur + 1) % 3], kPullsEnd);
        const bool pull = P > p.pull_min && !large;  // grid-uniform
        const int buf = cur & 1, ob = (cur + 1) & 1;
        if (gtid == 0) trace_round(p.trace, iters, (long long)P, pull ? 1 : 0);
        if (F == 0 && D == 0) break;
        // end of an epoch: the state rests in the arrays for the next one
        if (p.epoch_rounds > 0 && iters >= p.epoch_rounds) break;
        if (++iters > p.max_iter) {
            // Round cap: activated lanes keep their residual (never popped); their
            // activity masks are cleared for the next launch.
            if (gtid == 0) atomicOr(flags, C2G_FLAG_ITER_CAP);
            for (unsigned j = gwarp; j < F; j += nwarps) {
                const int vw = ldcg(p.q[buf] + j).x;
                const unsigned lanes = ldcg(p.qmask[buf] + j);
                const size_t off = (size_t)(vw >> p.logW) * p.Q + ((vw & (W - 1)) << 5) + lane;
                if ((lanes >> lane) & 1u) p.res[off] = ldcg(p.rq[buf] + off) / one_m_a;
                if (lane == 0) p.amask[buf][vw] = 0u;
            }
            for (unsigned j = gwarp; j < D; j += nwarps)
                if (lane == 0) p.dmask[ldcg(p.dangle + j).x] = 0u;
            break;
        }
        // Pop the activated lanes without out-edges.
        for (unsigned j = gwarp; j < D; j += nwarps) {
            const int2 dv = ldcg(p.dangle + j);
            const size_t off = (size_t)(dv.x >> p.logW) * p.Q + ((dv.x & (W - 1)) << 5) + lane;
            if (((unsigned)dv.y >> lane) & 1u) p.res[off] = 0.0;
            if (lane == 0) p.dmask[dv.x] = 0u;
        }
        if (F == 0) break;
        // A pull round applies targets while it pulls: the pops above (residuals) and the
        // dangling list they read (which the applies refill) must be done first.
        if (pull && D > 0 && !grid_sync(bar, flags, p.barrier_ns)) return;
        if (F > p.qcap || ((T + (1u << kBatchTileLog) - 1u) >> kBatchTileLog) > p.mark_cap) {
            if (gtid == 0) atomicOr(flags, C2G_FLAG_BOUNDS);
            break;
        }
        const int nslot = (cur + 1) % 3, fslot = (cur + 2) % 3;
        if (gtid == 0) {
            ctl->qctr[fslot] = 0ull;
            ctl->dctr[fslot] = 0u;
            ctl->tilectr[fslot] = 0u;
            ctl->listctr[fslot] = 0u;
            ctl->pcount[fslot] = 0ull;
            ctl->popped += F;
            ctl->relaxed += T;
        }
        if (pull) {
            // Pull round, phase A: gather and sum the messages per target, and apply the
            // targets whose in-edges lie in one tile.
            if (gtid == 0) {
                pushes += (long long)P;
                steps += T;
            }
            touched += pbatch_pull<WP, LG>(p, buf, ob, &ctl->tilectr[cur % 3], psm, fst, pbatch_out(p, ob, nslot),
                                   &ctl->dctr[nslot], &ctl->listctr[cur % 3], psum, lane, bad);
        } else {
            // Push round, phase A: push along the frontier's edges (owner runs, as in the
            // SSSP batch): red.add of the FP64 message per active lane, red.or of the
            // word's sending lanes into the target's touched mask.
            const int2* q = p.q[buf];
            const unsigned* qm = p.qmask[buf];
            const int* mark = p.mark[buf];
            const double* rqb = p.rq[buf];
            const int tl = batch_tile_log(T, nwarps, kPushTileBig, kPushTileMin);
            const unsigned tile = 1u << tl;
            const unsigned ntiles = (T + tile - 1) >> tl;
            unsigned* tctr = &ctl->tilectr[cur % 3];
            unsigned tn = next_tile(tctr, lane);
            for (unsigned t = tn; t < ntiles; t = tn) {
                tn = next_tile(tctr, lane);  // the next tile, fetched while this one runs
                unsigned e0 = t << tl;
                const unsigned e1 = min(e0 + tile, T);
                unsigned o = (unsigned)ldcg(mark + (t << (tl - kBatchTileLog)));
                while (e0 < e1) {
                    const unsigned j = o + (unsigned)lane;
                    unsigned base = 0x7fffffffu, endv = 0xffffffffu, msk = 0u, rs = 0u;
                    int vw = 0;
                    bool badj = false;
                    if (j < F) {
                        const int2 qe = ldcg(q + j);
                        vw = qe.x;
                        base = (unsigned)qe.y;
                        const int v = vw >> p.logW;
                        rs = (unsigned)__ldg(p.row + v);
                        const unsigned deg = (unsigned)__ldg(p.row + v + 1) - rs;
                        endv = base + deg;
                        badj = rs + deg > p.E || deg == 0u;
                        msk = ldcg(qm + j);
                    }
                    const unsigned seg_end = min(e1, (unsigned)__shfl_sync(kFull, endv, 31));
                    if (__any_sync(kFull, badj) || seg_end <= e0 || o >= F ||
                        (unsigned)__shfl_sync(kFull, (int)base, 0) > e0) {
                        if (lane == 0) atomicOr(flags, C2G_FLAG_BOUNDS);
                        break;
                    }
                    for (int k = 0; k < 32; ++k) {
                        const unsigned kb = (unsigned)__shfl_sync(kFull, (int)base, k);
                        if (kb >= seg_end) break;
                        const unsigned ke = (unsigned)__shfl_sync(kFull, (int)endv, k);
                        const unsigned lo = max(e0, kb), hi = min(seg_end, ke);
                        if (lo >= hi) continue;
                        const int kvw = __shfl_sync(kFull, vw, k);
                        const unsigned km = (unsigned)__shfl_sync(kFull, (int)msk, k);
                        const unsigned krs = (unsigned)__shfl_sync(kFull, (int)rs, k);
                        const unsigned w = (unsigned)kvw & (unsigned)(W - 1);
                        const unsigned cnt = (unsigned)__popc(km);
                        // slot -> query position of the word's active queries
                        if ((km >> lane) & 1u) qtab[__popc(km & ((1u << lane) - 1u))] = lane;
                        __syncwarp();
                        const int qp = (unsigned)lane < cnt ? qtab[lane] : 0;
                        __syncwarp();
                        double* mw = p.msg + (w << 5);  // + v * Q + query position
                        unsigned* trow = p.tmask + w;   // + (v << logW): touched word of v
                        // (1-alpha)*r_u of slot `lane`'s query, stored by the apply that
                        // activated it (src/ppr/purn/Main.cu:288)
                        const double qu = (unsigned)lane < cnt
                                              ? ldcg(rqb + (size_t)((unsigned)kvw >> p.logW) * Qu + (w << 5) + qp)
                                              : 0.0;
                        const DSplit qs = c2g_dsplit(qu);
                        // exponent and high significand in one word (0: residual outside the
                        // integer product's range, multiply on the FP64 pipe)
                        const unsigned qpk = c2g_mul_q_ok(qs) ? ((unsigned)qs.e << 21) | qs.hi : 0u;
                        const unsigned len = hi - lo;
                        const int2* eadj = p.adj + krs + (lo - kb);
                        owner_items<kPprBatchUnroll>(cnt, len, lane, [&](const int* eis, const int* js) {
                            int2 ew[kPprBatchUnroll];
                            bool ok[kPprBatchUnroll];
#pragma unroll
                            for (int u = 0; u < kPprBatchUnroll; ++u) {
                                ok[u] = (unsigned)eis[u] < len;
                                ew[u] = ok[u] ? __ldg(eadj + eis[u]) : make_int2(0, 0);
                            }
#pragma unroll
                            for (int u = 0; u < kPprBatchUnroll; ++u) {
                                const unsigned pk = (unsigned)__shfl_sync(kFull, (int)qpk, js[u]);
                                DSplit sj;
                                sj.lo = (unsigned)__shfl_sync(kFull, (int)qs.lo, js[u]);
                                sj.hi = pk & 0x1fffffu;
                                sj.e = (int)(pk >> 21);
                                const int qq = __shfl_sync(kFull, qp, js[u]);
                                const unsigned wb = (unsigned)ew[u].y;
                                // m = qu * w in FP64, on the integer pipes (fp64_mul.h)
                                bool send = ok[u] && (int)wb > 0;
                                const bool mok = pk != 0u && c2g_mul_w_ok(wb);
                                double m = c2g_mul(sj, wb);
                                const bool slow = __any_sync(kFull, send && !mok);
                                if (slow) {  // w subnormal: FP64 pipe
                                    const double quj = __shfl_sync(kFull, qu, js[u]);
                                    if (!mok) m = quj * (double)__uint_as_float(wb);
                                    send = send && (mok || m > 0.0);
                                }
                                const size_t tv = (size_t)(unsigned)ew[u].x;
                                if (send) atomicAdd(mw + tv * Qu + qq, m);
                                // Touched lanes: every active query sends along a positive
                                // weight, so slot 0 marks the whole word at once.
                                if (!slow) {
                                    if (send && js[u] == 0) atomicOr(trow + (tv << p.logW), km);
                                } else if (send) {
                                    atomicOr(trow + (tv << p.logW), 1u << qq);
                                }
                            }
                        });
                        if (lane == 0) pushes += (long long)cnt * len;
                        steps += len;
                    }
                    e0 = seg_end;
                    o += 32;
                }
            }
        }
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        phase_mark(ctl->phase_ns, tph, 2);
        if (gtid == 0) trace_mid(p.trace, iters - 1);
        // The frontier just consumed leaves the pull lookup.
        for (unsigned j = gtid; j < F; j += nthreads) p.amask[buf][ldcg(p.q[buf] + j).x] = 0u;
        // Phase B: apply the messages of the touched pairs and activate: after a pull, the
        // listed straddlers (unless the list overflowed); after a push, every touched word.
        const unsigned nl = pull ? ldcg(&ctl->listctr[cur % 3]) : 0u;
        const bool listed = pull && nl <= p.slist_cap;  // grid-uniform
        touched += pbatch_sweep<WP>(p, false, ob, listed ? p.slist : nullptr, nl, fst, pbatch_out(p, ob, nslot),
                                &ctl->dctr[nslot], psum, gwarp, nwarps, lane);
        if (lane == 0 && psum) atomicAdd(&ctl->pcount[nslot], psum);
        psum = 0;
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        phase_mark(ctl->phase_ns, tph, 1);
        ++cur;
    }
    if (bad) atomicOr(flags, C2G_FLAG_BOUNDS);
    // pushes are counted by lane 0 of each warp; touched lanes by every lane
    unsigned long long tl = touched;
    for (int o = 16; o >= 1; o >>= 1) tl += __shfl_xor_sync(kFull, tl, o);
    if (lane == 0) {
        atomicAdd((unsigned long long*)&p.counters[0], (unsigned long long)pushes);
        atomicAdd((unsigned long long*)&p.counters[1], (unsigned long long)steps);
        atomicAdd((unsigned long long*)&ctl->touched, tl);
    }
    if (gtid == 0) {
        ctl->iterations = iters;
        trace_round(p.trace, iters, 0, -1);
    }
}

// [V][Q] float -> caller layout (first nq queries).
__global__ void batch_transpose_f(const float* __restrict__ src, int V, int Q, int nq, float* __restrict__ out,
                                  int query_major) {
    const size_t total = (size_t)V * (size_t)nq;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        if (query_major) {
            const size_t qi = i / (size_t)V, v = i % (size_t)V;
            out[i] = src[v * Q + qi];
        } else {
            const size_t v = i / (size_t)nq, qi = i % (size_t)nq;
            out[i] = src[v * Q + qi];
        }
    }
}

// [V][Q] double -> caller layout as float (first nq queries).
__global__ void batch_transpose_d2f(const double* __restrict__ src, int V, int Q, int nq, float* __restrict__ out,
                                    int query_major) {
    const size_t total = (size_t)V * (size_t)nq;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        if (query_major) {
            const size_t qi = i / (size_t)V, v = i % (size_t)V;
            out[i] = (float)src[v * Q + qi];
        } else {
            const size_t v = i / (size_t)nq, qi = i % (size_t)nq;
            out[i] = (float)src[v * Q + qi];
        }
    }
}

// The kernel for queries in the first nq of 32 * 2^logW slots, with its shared memory allowed, its groups of query
// words and its blocks per SM.  Pulls take as many words at a time as hold queries: a resident batch of 64 slots
// with 11 queries at work pulls one word, not two (a wave of 32 mixed requests, scale 18: 27.5 -> 24.2 ms).
static int ppr_batch_kernel(int nq, const void** kernel, unsigned* groups, int* per_sm) {
    const unsigned words = ((unsigned)nq + 31u) / 32u;
    *groups = words <= 2u ? 1u : (words + 3u) / 4u;
    *kernel = words <= 1u ? nq <= 8    ? (const void*)ppr_batch_persistent<1, 4>
                            : nq <= 16 ? (const void*)ppr_batch_persistent<1, 8>
                                       : (const void*)ppr_batch_persistent<1, 16>
            : words == 2u ? (const void*)ppr_batch_persistent<2, 32>
                          : (const void*)ppr_batch_persistent<4, 32>;
    C2G_CUDA(cudaFuncSetAttribute(*kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPprBatchSmem));
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, *kernel, kPprBatchThreads, kPprBatchSmem));
    if (*per_sm < 1) return fail(C2G_ERR_CUDA, "batch kernel cannot be resident");
    return C2G_OK;
}

// log2 of the chunks of 32 in-edges per pull item: 8 chunks (a fourth of the rows then crosses an item
// boundary), fewer where that leaves the grid's warps less than 16 items each to level the round's
// end (40 queries at scale 16, 6 chunks per warp: 8-chunk items 14.8 ms a batch, 2 12.8, 1 11.7).  What
// is uneven is the chunks of a skewed graph: 32 rows of one in-edge, each an apply, or part of one hub's.  Where no row
// has more than 256 in-edges (no segments) 3 items per warp are enough, and shorter items would only cut rows: 4M
// edges on 100,000 uniform vertices, 70 queries 14.0 ms a batch with 1 chunk per item, 9.6 with 4 or 8, 250 queries
// 41.8 / 23.4 / 21.6; 2M on 250,000, 130 queries 30.8 / 26.7 / 26.9.
static int ppr_pull_log(const c2g_graph* g, unsigned groups, int blocks) {
    const size_t chunks = ((size_t)g->E + 31) / 32, warps = (size_t)blocks * (kPprBatchThreads / 32);
    int k = 3;
    while (k > 0 && (chunks >> k) * groups < (g->rows_in.n[0] ? 16 : 3) * warps) --k;
    return k;
}

struct PprBatchWork {
    float* pr = nullptr;
    double* res = nullptr;
    double* msg = nullptr;
    double* rq = nullptr;
    double* rq2 = nullptr;
    float2* rqf[2] = {nullptr, nullptr};
    unsigned* amask[2] = {nullptr, nullptr};
    unsigned* tmask = nullptr;
    unsigned* slist = nullptr;
    unsigned slist_cap = 0;
    unsigned* dmask = nullptr;
    int2* q[2] = {nullptr, nullptr};
    unsigned* qmask[2] = {nullptr, nullptr};
    int* mark[2] = {nullptr, nullptr};
    int2* dangle = nullptr;
    TraversalCtl* ctl = nullptr;
    long long* counters = nullptr;
    int* src = nullptr;
    int* seed_off = nullptr;
    int* seed_v = nullptr;
    float* seed_w = nullptr;
    float* stage = nullptr;
    RoundTrace* trace = nullptr;
    size_t seed_cap = 0;
    int Q = 0;
    bool clean = false;  // msg, tmask and amask are zero
};

void ppr_batch_free(c2g_graph* g) {
    PprBatchWork* w = reinterpret_cast<PprBatchWork*>(g->ppr_batch);
    if (!w) return;
    if (g->last_trace == w->trace) g->last_trace = nullptr;
    void* ptrs[] = {w->pr, w->res, w->msg, w->rq, w->rq2, w->rqf[0], w->rqf[1], w->amask[0], w->amask[1], w->tmask,
                    w->slist, w->dmask,
                    w->q[0], w->q[1],
                    w->qmask[0], w->qmask[1],
                    w->mark[0], w->mark[1], w->dangle, w->ctl, w->counters, w->src, w->seed_off,
                    w->seed_v, w->seed_w, w->stage, w->trace};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete w;
    g->ppr_batch = nullptr;
}

static int ppr_batch_alloc(c2g_graph* g, int Q, size_t n_seeds) {
    PprBatchWork* w = reinterpret_cast<PprBatchWork*>(g->ppr_batch);
    if (w && w->Q >= Q && w->seed_cap >= n_seeds) return C2G_OK;
    if (w) ppr_batch_free(g);
    w = new PprBatchWork();
    g->ppr_batch = w;
    const size_t V = g->V ? (size_t)g->V : 1;
    const size_t W = (size_t)Q / 32, VQ = V * (size_t)Q;
    const size_t qcap = V * W;
    const size_t mark_cap = (((size_t)g->E * W) >> kBatchTileLog) + 2;
    C2G_CUDA(cudaMalloc(&w->pr, sizeof(float) * VQ));
    C2G_CUDA(cudaMalloc(&w->res, sizeof(double) * VQ));
    C2G_CUDA(cudaMalloc(&w->msg, sizeof(double) * VQ));
    C2G_CUDA(cudaMalloc(&w->rq, sizeof(double) * VQ));
    C2G_CUDA(cudaMalloc(&w->rq2, sizeof(double) * VQ));
    C2G_CUDA(cudaMalloc(&w->rqf[0], sizeof(float2) * VQ));
    C2G_CUDA(cudaMalloc(&w->rqf[1], sizeof(float2) * VQ));
    C2G_CUDA(cudaMalloc(&w->tmask, sizeof(unsigned) * qcap));
    // pull rounds' straddlers: at most one owner per chunk boundary, W words each
    w->slist_cap = (unsigned)std::min(qcap, (((size_t)g->E >> 5) + 1) * W);
    C2G_CUDA(cudaMalloc(&w->slist, sizeof(unsigned) * w->slist_cap));
    C2G_CUDA(cudaMalloc(&w->dmask, sizeof(unsigned) * qcap));
    C2G_CUDA(cudaMalloc(&w->amask[0], sizeof(unsigned) * qcap));
    C2G_CUDA(cudaMalloc(&w->amask[1], sizeof(unsigned) * qcap));
    for (int b = 0; b < 2; ++b) {
        C2G_CUDA(cudaMalloc(&w->q[b], sizeof(int2) * qcap));
        C2G_CUDA(cudaMalloc(&w->qmask[b], sizeof(unsigned) * qcap));
        C2G_CUDA(cudaMalloc(&w->mark[b], sizeof(int) * mark_cap));
    }
    C2G_CUDA(cudaMalloc(&w->dangle, sizeof(int2) * qcap));
    C2G_CUDA(cudaMalloc(&w->ctl, sizeof(TraversalCtl)));
    C2G_CUDA(cudaMalloc(&w->counters, sizeof(long long) * 2));
    C2G_CUDA(cudaMalloc(&w->src, sizeof(int) * (size_t)Q));
    C2G_CUDA(cudaMalloc(&w->seed_off, sizeof(int) * ((size_t)Q + 1)));
    w->seed_cap = n_seeds > 0 ? n_seeds : 1;
    C2G_CUDA(cudaMalloc(&w->seed_v, sizeof(int) * w->seed_cap));
    C2G_CUDA(cudaMalloc(&w->seed_w, sizeof(float) * w->seed_cap));
    C2G_CUDA(cudaMalloc(&w->trace, sizeof(RoundTrace) * (kMaxTraceRounds + 1)));
    w->Q = Q;
    w->clean = false;
    return C2G_OK;
}

// Largest positive weight of the reverse CSR (its bits: positive floats order as
// integers).  From 2^30 on, infinity and NaN included, pull rounds are off.
__global__ void weight_stats_kernel(const int2* __restrict__ adj_r, long long E, unsigned* wmax_bits) {
    unsigned wm = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < E; e += (long long)gridDim.x * blockDim.x) {
        const int wb = __ldg(adj_r + e).y;
        if (wb > 0) wm = max(wm, (unsigned)wb);
    }
    for (int o = 16; o >= 1; o >>= 1) wm = max(wm, (unsigned)__shfl_xor_sync(kFull, (int)wm, o));
    if ((threadIdx.x & 31) == 0 && wm) atomicMax(wmax_bits, wm);
}

// Reverse CSR and weight statistics for pull rounds (once per graph and weights).
int ppr_pull_prepare(c2g_graph* g) {
    int rc = build_reverse_graph(g);
    if (rc || g->wstat_valid) return rc;
    unsigned* d = nullptr;
    C2G_CUDA(cudaMalloc(&d, sizeof(unsigned)));
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(unsigned), g->stream);
    if (e == cudaSuccess && g->E > 0) {
        weight_stats_kernel<<<g->num_sms * 8, 256, 0, g->stream>>>(g->adj_r, (long long)g->E, d);
        e = cudaGetLastError();
    }
    unsigned h = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    cudaFree(d);
    C2G_CUDA(e);
    g->wstat_wmax_bits = h;
    g->wstat_valid = true;
    return C2G_OK;
}

// Push count above which a round pulls (c2g_ppr_batch_set_pull): pull rounds need the
// reverse CSR (a view uses its base's, never builds it) and weights below 2^30; with rmax
// below 1e-30 pushed residuals may leave the FP32 range of the pull's float pairs, so such
// launches push only.
//
// At the default ratio: 8 E, but for a batch of nq queries (0: a resident batch, whose slots say little
// about the queries at work) half an E per query for fewer than 16, and E / 4 for up to 64 on
// graphs up to kSmallPullEdges, where a round is latency and a pull saves the push's atomics and its sweep.  ms a batch
// at 8 E / this: 5 queries at scale 14 7.39 / 3.95, 2 6.74 / 3.74, 20 4.82 / 4.57, 3 on 3,000 uniform
// vertices 5.48 / 2.30, 4 at scale 18 10.4 / 9.5, 8 11.6 / 10.1, 3 at scale 20 27.5 / 25.2; 11 or more at scale
// 18 are within 1%; 250 on 100,003 uniform vertices 35.9 at 8 E, 37.4 at E / 4.
constexpr int64_t kSmallPullEdges = 1 << 20;

static int ppr_pull_threshold(c2g_graph* g, const c2g_ppr_params& prm, int nq, unsigned long long* pull_min) {
    *pull_min = ~0ull;
    float ratio = g->ppr_cfg.batch_pull_ratio;
    if (ratio == kDefaultPullRatio && nq > 0)
        ratio = nq <= 64 && g->E <= kSmallPullEdges ? 0.25f : std::min(ratio, 0.5f * (float)nq);
    if (ratio >= 0.f && g->E > 0 && prm.rmax >= 1e-30f && (g->wstat_valid || !g->borrowed)) {
        int rc;
        if (!g->borrowed && (rc = ppr_pull_prepare(g))) return rc;
        if (g->wstat_wmax_bits < kPullMaxWeight) *pull_min = (unsigned long long)((double)ratio * (double)g->E);
    }
    return C2G_OK;
}

// msg, tmask, dmask and both activity masks are zero between launches.
static int ppr_batch_clean(c2g_graph* g, PprBatchWork* w) {
    if (w->clean) return C2G_OK;
    const size_t VQ = (size_t)g->V * (size_t)w->Q;
    C2G_CUDA(cudaMemsetAsync(w->msg, 0, sizeof(double) * VQ, g->stream));
    for (unsigned* m : {w->tmask, w->dmask, w->amask[0], w->amask[1]})
        C2G_CUDA(cudaMemsetAsync(m, 0, sizeof(unsigned) * (size_t)g->V * (size_t)(w->Q / 32), g->stream));
    w->clean = true;
    return C2G_OK;
}

static void ppr_batch_params(c2g_graph* g, PprBatchWork* w, int Q, int logW, const c2g_ppr_params& prm,
                             unsigned long long pull_min, PprBatchParams& p) {
    const int nq = Q;
    const std::vector<int32_t>* seed_off = nullptr;
    p.row = g->row;
    p.adj = g->adj_f;
    p.E = (unsigned)g->E;
    p.V = g->V;
    p.logW = logW;
    p.Q = Q;
    p.nq = nq;
    p.pr = w->pr;
    p.res = w->res;
    p.msg = w->msg;
    p.rq[0] = w->rq;
    p.rq[1] = w->rq2;
    p.amask[0] = w->amask[0];
    p.amask[1] = w->amask[1];
    p.rqf[0] = w->rqf[0];
    p.rqf[1] = w->rqf[1];
    p.tmask = w->tmask;
    p.slist = w->slist;
    p.slist_cap = w->slist_cap;
    p.dmask = w->dmask;
    p.epoch_rounds = 0;
    p.cur0 = 1;
    for (int b = 0; b < 2; ++b) {
        p.q[b] = w->q[b];
        p.qmask[b] = w->qmask[b];
        p.mark[b] = w->mark[b];
    }
    p.dangle = w->dangle;
    p.ctl = w->ctl;
    p.sources = w->src;
    p.seed_off = seed_off ? w->seed_off : nullptr;
    p.seed_v = w->seed_v;
    p.seed_w = w->seed_w;
    p.alpha = prm.alpha;
    p.rmax = prm.rmax;
    p.r0 = prm.r0;
    p.pr0 = prm.pr0;
    p.seeded = prm.seeded;
    p.max_iter = prm.max_iter;
    p.qcap = (unsigned)((size_t)g->V * (size_t)(p.Q / 32));
    p.mark_cap = (unsigned)((((size_t)g->E * (size_t)(p.Q / 32)) >> kBatchTileLog) + 2);
    p.barrier_ns = g->barrier_ns ? g->barrier_ns : 4000000000ull;
    p.counters = w->counters;
    p.adj_r = g->adj_r;
    p.r_bits = g->r_bits;
    p.r_prefix = g->r_prefix;
    p.r_rows = g->r_rows;
    p.pull_log = 3;
    p.pull_min = pull_min;
    p.trace = w->trace;
    g->last_trace = w->trace;
}

int ppr_batch_launch(c2g_graph* g, int32_t nq, const int32_t* sources, const c2g_ppr_params& prm,
                     const std::vector<int32_t>* seed_off, const std::vector<int32_t>* seed_v,
                     const std::vector<float>* seed_w, float* pr_out, float* res_out, int on_device, int query_major,
                     float* ms, long long* counters, TraversalCtl* ctl_out) {
    if (!g->adj_f) return fail(C2G_ERR_UNSUPPORTED, "graph has no float weights (flist / ppr wlist)");
    int Q = 32, logW = 0;
    while (Q < nq) {
        Q <<= 1;
        ++logW;
    }
    if ((size_t)g->V * (size_t)(Q / 32) >= (size_t(1) << 31) || (size_t)g->E * (size_t)(Q / 32) >= (size_t(1) << 32))
        return fail(C2G_ERR_RANGE, "batch of %d queries too large for this graph", nq);
    int rc;
    const size_t ns = seed_v ? seed_v->size() : 0;
    unsigned long long pull_min = ~0ull;
    if ((rc = ppr_pull_threshold(g, prm, nq, &pull_min))) return rc;
    if ((rc = ppr_batch_alloc(g, Q, ns))) return rc;
    PprBatchWork* w = reinterpret_cast<PprBatchWork*>(g->ppr_batch);
    int coop = 0, per_sm = 0;
    const void* kernel = nullptr;
    C2G_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g->device));
    if (!coop) return fail(C2G_ERR_UNSUPPORTED, "device lacks cooperative launch");
    unsigned groups = 0;
    if ((rc = ppr_batch_kernel(nq, &kernel, &groups, &per_sm))) return rc;
    const size_t VQ = (size_t)g->V * (size_t)w->Q;
    if ((rc = ppr_batch_clean(g, w))) return rc;
    C2G_CUDA(cudaMemcpyAsync(w->src, sources, sizeof(int) * (size_t)nq, cudaMemcpyHostToDevice, g->stream));
    if (seed_off) {
        C2G_CUDA(cudaMemcpyAsync(w->seed_off, seed_off->data(), sizeof(int) * seed_off->size(), cudaMemcpyHostToDevice,
                                 g->stream));
        if (ns) {
            C2G_CUDA(cudaMemcpyAsync(w->seed_v, seed_v->data(), sizeof(int) * ns, cudaMemcpyHostToDevice, g->stream));
            C2G_CUDA(cudaMemcpyAsync(w->seed_w, seed_w->data(), sizeof(float) * ns, cudaMemcpyHostToDevice, g->stream));
        }
    }
    PprBatchParams p;
    ppr_batch_params(g, w, Q, logW, prm, pull_min, p);
    p.nq = nq;
    p.seed_off = seed_off ? w->seed_off : nullptr;
    const int blocks = grid_blocks(g, per_sm);
    p.pull_groups = groups;
    p.pull_log = ppr_pull_log(g, groups, blocks);
    C2G_CUDA(cudaMemsetAsync(w->ctl, 0, sizeof(TraversalCtl), g->stream));
    C2G_CUDA(cudaMemsetAsync(w->counters, 0, sizeof(long long) * 2, g->stream));
    void* args[] = {&p};
    C2G_CUDA(cudaEventRecord(g->ev0, g->stream));
    C2G_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(kPprBatchThreads), args, kPprBatchSmem, g->stream));
    C2G_CUDA(cudaEventRecord(g->ev1, g->stream));
    cudaError_t e = cudaSuccess;
    float* outs[2] = {pr_out, res_out};
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
        if (!outs[k]) continue;
        float* dst = outs[k];
        float* direct = on_device ? nullptr : static_cast<float*>(mapped_host(outs[k]));
        if (direct) {
            dst = direct;
        } else if (!on_device) {
            if (!w->stage) e = cudaMalloc(&w->stage, sizeof(float) * VQ);
            dst = w->stage;
        }
        if (e != cudaSuccess) break;
        if (k == 0)
            if (query_major)
                launch_transpose_qmajor<float, float>(w->pr, g->V, p.Q, nq, dst, g->stream);
            else
                batch_transpose_f<<<g->num_sms * 8, 256, 0, g->stream>>>(w->pr, g->V, p.Q, nq, dst, query_major);
        else
            if (query_major)
                launch_transpose_qmajor<double, float>(w->res, g->V, p.Q, nq, dst, g->stream);
            else
                batch_transpose_d2f<<<g->num_sms * 8, 256, 0, g->stream>>>(w->res, g->V, p.Q, nq, dst, query_major);
        e = cudaGetLastError();
        if (e == cudaSuccess && !on_device && !direct)
            e = cudaMemcpyAsync(outs[k], dst, sizeof(float) * (size_t)g->V * (size_t)nq, cudaMemcpyDeviceToHost,
                                g->stream);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctl_out, w->ctl, sizeof(TraversalCtl), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(counters, w->counters, sizeof(long long) * 2, cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    C2G_CUDA(e);
    if (ctl_out->flags & (C2G_FLAG_BARRIER_TIMEOUT | C2G_FLAG_QUEUE_OVERFLOW | C2G_FLAG_BOUNDS)) w->clean = false;
    C2G_CUDA(cudaEventElapsedTime(ms, g->ev0, g->ev1));
    return C2G_OK;
}

// Resident batch (c2g_session): the workspace of Q query slots with every array at rest
// (pr, res, msg and the masks zero), its arrays, and one epoch of at most `rounds` rounds
// starting at round cur0 from the state the previous epoch (and the joins since) left.
int ppr_batch_reserve(c2g_graph* g, int Q, PprBatchArrays* a) {
    if (!g->adj_f) return fail(C2G_ERR_UNSUPPORTED, "graph has no float weights (flist / ppr wlist)");
    if ((size_t)g->V * (size_t)(Q / 32) >= (size_t(1) << 31) || (size_t)g->E * (size_t)(Q / 32) >= (size_t(1) << 32))
        return fail(C2G_ERR_RANGE, "%d slots too many for this graph", Q);
    int rc;
    if ((rc = ppr_batch_alloc(g, Q, 0))) return rc;
    PprBatchWork* w = reinterpret_cast<PprBatchWork*>(g->ppr_batch);
    w->clean = false;
    if ((rc = ppr_batch_clean(g, w))) return rc;
    const size_t VQ = (size_t)g->V * (size_t)w->Q;
    C2G_CUDA(cudaMemsetAsync(w->pr, 0, sizeof(float) * VQ, g->stream));
    C2G_CUDA(cudaMemsetAsync(w->res, 0, sizeof(double) * VQ, g->stream));
    C2G_CUDA(cudaStreamSynchronize(g->stream));
    a->pr = w->pr;
    a->res = w->res;
    a->rq[0] = w->rq;
    a->rq[1] = w->rq2;
    a->rqf[0] = w->rqf[0];
    a->rqf[1] = w->rqf[1];
    a->amask[0] = w->amask[0];
    a->amask[1] = w->amask[1];
    a->dmask = w->dmask;
    return C2G_OK;
}

int ppr_batch_epoch(c2g_graph* g, int Q, int used, const c2g_ppr_params& prm, int cur0, int rounds, float* ms,
                    long long* counters, TraversalCtl* ctl_out) {
    PprBatchWork* w = reinterpret_cast<PprBatchWork*>(g->ppr_batch);
    if (!w || w->Q < Q) return fail(C2G_ERR_ARG, "resident PPR batch has no workspace");
    int logW = 0;
    while ((32 << logW) < Q) ++logW;
    int rc;
    unsigned long long pull_min = ~0ull;
    if ((rc = ppr_pull_threshold(g, prm, 0, &pull_min))) return rc;  // slots, not queries
    int per_sm = 0;
    const void* kernel = nullptr;
    unsigned groups = 0;
    if ((rc = ppr_batch_kernel(used, &kernel, &groups, &per_sm))) return rc;
    PprBatchParams p;
    ppr_batch_params(g, w, Q, logW, prm, pull_min, p);
    const int blocks = grid_blocks(g, per_sm);
    p.pull_groups = groups;
    p.pull_log = ppr_pull_log(g, groups, blocks);
    p.epoch_rounds = rounds < 1 ? 1 : rounds;
    p.cur0 = cur0;
    p.max_iter = 1 << 30;  // the per-query caps are the session's
    C2G_CUDA(cudaMemsetAsync(w->ctl, 0, sizeof(TraversalCtl), g->stream));
    C2G_CUDA(cudaMemsetAsync(w->counters, 0, sizeof(long long) * 2, g->stream));
    void* args[] = {&p};
    C2G_CUDA(cudaEventRecord(g->ev0, g->stream));
    C2G_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(kPprBatchThreads), args, kPprBatchSmem, g->stream));
    C2G_CUDA(cudaEventRecord(g->ev1, g->stream));
    C2G_CUDA(cudaMemcpyAsync(ctl_out, w->ctl, sizeof(TraversalCtl), cudaMemcpyDeviceToHost, g->stream));
    C2G_CUDA(cudaMemcpyAsync(counters, w->counters, sizeof(long long) * 2, cudaMemcpyDeviceToHost, g->stream));
    C2G_CUDA(cudaStreamSynchronize(g->stream));
    C2G_CUDA(cudaEventElapsedTime(ms, g->ev0, g->ev1));
    return C2G_OK;
}

}  // namespace c2g
