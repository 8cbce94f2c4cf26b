// Single-query forward push (PPR and the reference's adsorption variant) for sm_103a:
// one persistent cooperative launch per query.
//
// Replaces calcuatePPR (reference src/ppr/base/Main.cu:122-395, src/ppr/purn/Main.cu:
// 149-428, src/adsorption/w-base/Main.cu:124-395) with the same BSP semantics:
//   round: every frontier vertex u pushes (1-alpha)*r_u*w(u,v) into msg[v];
//   then every vertex v that got a message: res[v] += msg[v]; msg[v] = 0;
//        if res[v] > rmax: pr[v] += alpha*res[v] and v joins the next frontier.
//
// Precision: edge weights and pr are FP32; the residual state (res, msg, the residual that a push
// round pushes) is FP64.  Pull rounds take the pushed residuals as float pairs (cut to 47 bits) and sum their
// messages as float pairs before they meet the FP64 residual: over 40 drawn queries, batches and gradients the L1 error of
// each output against 64 bits is that of the all-FP64 push to six digits.  res > rmax is a threshold: FP32 residuals of vertices
// sitting at rmax land on the other side of it than FP64 ones, each such flip moves
// about rmax of mass and cascades downstream, so FP32 residual bookkeeping drifts past
// L1 1e-6 of the FP64 result as graphs grow.  With FP64 residuals the decisions match the
// FP64 push up to summation order and the pairs' 2^-47.
//
// Round shapes, chosen per round from the frontier's out-edge count T:
//   * push (T small): edge-tiled walk over the frontier's out-edges, FP64 atomicAdd into
//     msg; the add that returns 0 records the target in the touched list and phase B
//     visits only touched vertices (no O(V) sweep, src/ppr/purn/Main.cu:379-407); with more
//     edges the adds keep no list and phase B sweeps all vertices;
//   * pull (T large, or a small graph): every vertex with in-edges gathers the pushed residuals
//     of its in-neighbours from a dense array qf, sums the messages in registers and
//     applies them on the spot: no message array, no atomics, one barrier a round.
// All give the same BSP round.
// The residual a frontier vertex pushes is captured when it is activated (nothing
// changes it before its pop).  Activated vertices without out-edges sit in a side list
// whose residual is cleared at the start of the next round, which is when the reference
// pops them (when the round cap ends the run first, they keep it).
#include <algorithm>
#include <climits>

#include "device_common.cuh"
#include "fp64_mul.h"
#include "internal.h"

namespace c2g {

struct PprParams {
    const int* row;
    const int2* adj;  // (target, float weight bits)
    unsigned E;
    int V;
    const int* row_r;   // reverse CSR (in-edges carrying w(u,v)), or nullptr: push only
    const int2* adj_r;
    RowLists rows;      // its rows by length
    unsigned* arrived;  // class 0: segments of a row summed so far, zero between rounds
    unsigned pull_min;   // pull when T is larger (~0: never),
    unsigned pull_next;  // after a pull when it is larger than this
    bool one_step;      // every round pulls, and its row lists are at most one step per warp
    int dense_div;      // dense push round (no touched list) when T * dense_div > E (0: never)
    float* pr;
    double* res;
    double* msg;
    float2* qf[2];  // (1-alpha)*r of the frontier's vertices as a float pair, 0 elsewhere, by round parity (pulls)
    int* stamp;
    int2* q[2];
    double* qval[2];
    int* mark[2];
    int* touched;
    int* dangle;
    TraversalCtl* ctl;
    StampState* st;
    int source;
    float alpha, rmax, r0, pr0;
    float absorb;         // pr += absorb * r at activation (alpha for PPR, 1 for the adjoint)
    int n_src;            // base init over a list of distinct sources (adjoint targets)
    const int* src_list;  // nullptr: the single `source`
    const float* src_r0;
    int max_iter;
    int seeded;
    const int* seed_v;  // pruned records of the source (seeded mode)
    const float* seed_w;
    int n_rec;
    int log_tile;
    unsigned mark_cap;
    unsigned long long barrier_ns;
};

__device__ __forceinline__ FrontierOut ppr_out(const PprParams& p, int buf, int slot) {
    FrontierOut o;
    o.q = p.q[buf];
    o.val = nullptr;
    o.vald = p.qval[buf];
    o.mark = p.mark[buf];
    o.ctr = &p.ctl->qctr[slot];
    o.cap = (unsigned)p.V;
    o.mark_cap = p.mark_cap;
    o.log_tile = p.log_tile;
    o.flags = &p.ctl->flags;
    return o;
}

constexpr int kPprUnroll = 8;  // edges in flight per lane
constexpr int kPprThreads = 512;  // launch shape of the persistent push
constexpr int kPprBlocksPerSm = 2;
constexpr unsigned kStepsPerBlock = 2;  // steps of a small graph's pull that are worth another block
// Round-robin tiles in push rounds (a dynamic tile queue measured no faster: 20.2 vs 20.4 ms
// per scale-22 query).
constexpr bool kPprDynTiles = false;

// Push round, phase A.  The first message a vertex gets in a round is the one whose
// atomicAdd returns 0 (msg[v] is 0 between rounds and every message is positive), so no
// separate touched flag is needed.  Zero messages are dropped: a vertex outside the
// frontier never holds a residual above rmax, so a zero message cannot activate it.
// With track = false (a dense round) the adds are fire-and-forget red.add and the
// apply pass sweeps all vertices instead of a touched list.
__device__ __forceinline__ void ppr_push(const PprParams& p, int buf, int slot, unsigned F, unsigned T,
                                         WarpStage& tst, bool track) {
    constexpr int U = kPprUnroll;
    const double* qv = p.qval[buf];
    walk_frontier_edges<U>(
        p.q[buf], p.mark[buf], p.row, F, T, p.log_tile, p.mark_cap, (unsigned)p.V, p.E, &p.ctl->flags,
        // (1-alpha)*r_u (src/ppr/purn/Main.cu:288); the owner is popped, so it leaves qf
        [&](int v, unsigned j) {
            p.qf[buf][v] = make_float2(0.f, 0.f);
            return ldcg(qv + j);
        },
        [&](const bool* ok, const unsigned* idx, const double* qu) {
            int c[U];
            double m[U];
            bool send[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int2 ew = ok[u] ? __ldg(p.adj + idx[u]) : make_int2(0, 0);
                c[u] = ew.x;
                // m = qu * w in FP64, on the integer pipes (fp64_mul.h); a message is sent
                // when it is positive (w > 0: qu > 0 for every activated vertex)
                const unsigned wb = (unsigned)ew.y;
                const DSplit qs = c2g_dsplit(qu[u]);
                const bool mok = c2g_mul_q_ok(qs) && c2g_mul_w_ok(wb);
                send[u] = ok[u] && ew.y > 0;
                m[u] = c2g_mul(qs, wb);
                if (__any_sync(kFull, send[u] && !mok)) {  // w subnormal: FP64 pipe
                    if (!mok) m[u] = qu[u] * (double)__int_as_float(ew.y);
                    send[u] = send[u] && (mok || m[u] > 0.0);
                }
            }
            if (!track) {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (send[u]) atomicAdd(p.msg + c[u], m[u]);
                return;
            }
            unsigned long long old[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                old[u] = send[u] ? c2g_dbits(atomicAdd(p.msg + c[u], m[u])) : 1ull;
#pragma unroll
            for (int u = 0; u < U; ++u)
                list_stage_push(tst, p.touched, &p.ctl->listctr[slot], (unsigned)p.V, &p.ctl->flags,
                                old[u] == 0ull, c[u]);
        },
        kPprDynTiles ? &p.ctl->tilectr[slot] : nullptr);
    if (track) list_stage_flush(tst, p.touched, &p.ctl->listctr[slot], (unsigned)p.V, &p.ctl->flags);
}

// Pulls end when a pushed residual passes kPullMaxQ.  The rounds' word for it is kept by
// round slot like the counts: a round reads its own slot's and whoever finds such a residual writes the
// next round's, so nothing that a round reads is written while it runs (a pull round has one barrier, at its
// end).  A pull writes it beside the next round's counts (kPullsEnd in ctl->pcount: a load of its own costs a round of a
// million edges 3%), a push into ctl->farmin, where a round that finds it set hands it on, so that it stays.
constexpr unsigned long long kPullsEnd = 1ull << 63;
__device__ __forceinline__ unsigned pull_frontier(unsigned long long c) { return (unsigned)((c & ~kPullsEnd) >> 32); }

// The float pair of a pushed residual (fp64_mul.h), and its value.
__device__ __forceinline__ float2 ppr_pair(double q) {
    if (c2g_split_ok(q)) {
        const c2g_pair hl = c2g_split_pair(q);
        return make_float2(c2g_bitsf(hl.hi), c2g_bitsf(hl.lo));
    }
    const float hi = __double2float_rz(q);
    return make_float2(hi, __double2float_rz(q - (double)hi));
}
__device__ __forceinline__ double ppr_pair_value(const float2& q) {
    return c2g_float_bits_to_double(__float_as_uint(q.x)) + c2g_float_bits_to_double(__float_as_uint(q.y));
}

// Sum of two floats as a rounded sum and its error.
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
    const float s = __fadd_rn(a, b), bv = __fsub_rn(s, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bv)), __fsub_rn(b, bv));
    return s;
}

// Totals of a pull round: activated vertices with out-edges (F << 32 | their out-edges) and without.
struct PullTotals {
    unsigned long long count;
    unsigned dangling;
    int qmax;  // largest pushed residual (float bits)
};

// Pull round.  The rows of the reverse CSR are binned by length (RowLists), so that a warp takes 32 / L
// rows of similar length, L lanes each and at most kLaneEdges in-edges per lane: all its gathers
// are in flight together, and a row's sum is its lanes' messages and log2(L) shuffles.  Messages
// are summed as float pairs (products and sums with their errors recovered, about 47 bits
// relative, as in the batched push): a warp's FP64 instruction holds an SM's FP64 pipe for 16
// cycles here.  Rows of more than 256 edges are split into segments: each adds its sum to msg, and
// after one fence for all of a warp's segments the last segment of a row to arrive applies it
// (a fence per segment of 128 edges held a warp for a quarter of the round).
// A round over all 16M edges of a scale-20 graph takes 94 us; pushed, 240 us.
//
// qf[b] holds the frontier; the new one goes to qf[b ^ 1], for every row, so nothing is cleared.  A vertex
// that was in the frontier has residual 0 from its pop (its res still holds what it had when it was
// activated: at the round cap that is what it keeps); one that was not adds its messages to res.
struct PullSums {
    float hi, lo;
};

// s += q * w, exactly up to the last bits of lo; a source outside the frontier (q = 0) or a weight that is
// not positive adds 0.
__device__ __forceinline__ void pull_add(const float2& q, int wbits, PullSums& s) {
    const float w = q.x != 0.f ? __int_as_float(wbits) : 0.f;
    const float pm = __fmul_rn(q.x, w);
    const float pe = __fmaf_rn(q.y, w, __fmaf_rn(q.x, w, -pm));
    float te;
    s.hi = two_sum(s.hi, pm, te);
    s.lo = __fadd_rn(s.lo, __fadd_rn(te, pe));
}

// Messages of this lane's in-edges first, first + step, ... (up to kLaneEdges of them) below n.
__device__ __forceinline__ void pull_lane(const int2* __restrict__ adj, const float2* qin, int first, int step, int n,
                                          PullSums& s) {
    int2 ew[kLaneEdges];
    float2 q[kLaneEdges];
#pragma unroll
    for (int u = 0; u < kLaneEdges; ++u) {
        const int i = first + u * step;
        ew[u] = i < n ? __ldg(adj + i) : make_int2(0, 0);
    }
    // through L1: qf[b] does not change during the round
#pragma unroll
    for (int u = 0; u < kLaneEdges; ++u) q[u] = ew[u].y > 0 ? __ldca(qin + ew[u].x) : make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < kLaneEdges; ++u) pull_add(q[u], ew[u].y, s);
}

// Sum over groups of L lanes; the value as a double (in every lane of the group).
__device__ __forceinline__ double pull_reduce(PullSums s, int L) {
    for (int o = 1; o < L; o <<= 1) {
        const float oh = __shfl_xor_sync(kFull, s.hi, o), ol = __shfl_xor_sync(kFull, s.lo, o);
        float te;
        s.hi = two_sum(s.hi, oh, te);
        s.lo = __fadd_rn(te, __fadd_rn(s.lo, ol));
    }
    return ppr_pair_value(make_float2(s.hi, s.lo));
}

// Vertex v's messages s are complete (q0: the high half of its own pushed residual, r0: its res,
// pr0: its pr).
__device__ __forceinline__ void pull_apply(const PprParams& p, float2* qout, int v, int out_degree, double s, float q0,
                                           double r0, float pr0, PullTotals& tot) {
    const bool popped = q0 != 0.f;
    float2 q1 = make_float2(0.f, 0.f);
    if (c2g_dbits(s) != 0ull) {  // messages are positive
        const double r = popped ? s : r0 + s;
        p.res[v] = r;
        if (c2g_dbits(r) > c2g_dbits((double)p.rmax)) {  // both non-negative
            p.pr[v] = pr0 + (float)((double)p.absorb * r);
            q1 = ppr_pair((1.0 - (double)p.alpha) * r);
            tot.qmax = max(tot.qmax, __float_as_int(q1.x));
            if (out_degree > 0)
                tot.count += (1ull << 32) | (unsigned)out_degree;
            else
                ++tot.dangling;
        }
    } else if (popped) {
        p.res[v] = 0.0;
    }
    qout[v] = q1;
}

__device__ __forceinline__ void ppr_pull(const PprParams& p, int b, PullTotals& tot) {
    const int lane = threadIdx.x & 31;
    const unsigned gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
    const float2* qin = p.qf[b];
    float2* qout = p.qf[b ^ 1];
    const RowLists& R = p.rows;
    // segments of long rows
    for (unsigned r = gwarp; r < R.n[0]; r += nwarps) {
        const int4 rec = __ldg(R.rec + r);
        PullSums s{0.f, 0.f};
        for (int i = 0; i < rec.z; i += 32 * kLaneEdges)
            pull_lane(p.adj_r + rec.y, qin, i + lane, 32, rec.z, s);
        const double m = pull_reduce(s, 32);
        if (lane == 0 && c2g_dbits(m) != 0ull) atomicAdd(p.msg + rec.x, m);
    }
    if (gwarp < R.n[0]) {
        __syncwarp();
        __threadfence();  // the warp's sums are in msg before it arrives
        for (unsigned r0 = gwarp; r0 < R.n[0]; r0 += 32u * nwarps) {
            const unsigned r = r0 + (unsigned)lane * nwarps;
            if (r >= R.n[0]) continue;
            const int2 sg = __ldg(R.seg + r);
            if (atomicAdd(p.arrived + sg.x, 1u) != (unsigned)sg.y - 1u) continue;
            __threadfence();  // the other segments' sums are seen
            const int4 rec = __ldg(R.rec + r);
            const double m = ldcg(p.msg + rec.x);
            p.msg[rec.x] = 0.0;
            p.arrived[sg.x] = 0u;
            pull_apply(p, qout, rec.x, rec.w, m, ldcg(reinterpret_cast<const float*>(qin + rec.x)), ldcg(p.res + rec.x),
                       ldcg(p.pr + rec.x), tot);
        }
    }
    // whole rows, starting with the warps that had one segment less
    const unsigned units = R.unit[kRowClasses], turn = R.n[0] % nwarps;
    for (unsigned unit = R.unit[1] + (gwarp >= turn ? gwarp - turn : gwarp + nwarps - turn); unit < units;
         unit += nwarps) {
        int c = 1;
        unsigned n = R.n[1], off = R.off[1], first = R.unit[1];
#pragma unroll
        for (int k = 2; k < kRowClasses; ++k)
            if (unit >= R.unit[k]) {
                c = k;
                n = R.n[k];
                off = R.off[k];
                first = R.unit[k];
            }
        const int logL = 6 - c, L = 1 << logL, part = lane & (L - 1);
        const unsigned r = ((unit - first) << (5 - logL)) + (unsigned)(lane >> logL);
        const int4 rec = r < n ? __ldg(R.rec + off + r) : make_int4(0, 0, 0, 0);
        const bool mine = r < n && part == 0;
        float q0 = 0.f, pr0 = 0.f;
        double r0 = 0.0;
        if (mine) {
            q0 = ldcg(reinterpret_cast<const float*>(qin + rec.x));
            r0 = ldcg(p.res + rec.x);
            pr0 = ldcg(p.pr + rec.x);
        }
        PullSums s{0.f, 0.f};
        pull_lane(p.adj_r + rec.y, qin, part, L, rec.z, s);
        const double m = pull_reduce(s, L);
        if (mine) pull_apply(p, qout, rec.x, rec.w, m, q0, r0, pr0, tot);
    }
}

// A block's totals of a pull round join the next round's counts.
__device__ __forceinline__ void pull_totals(TraversalCtl* ctl, int nslot, PullTotals tot, PullTotals& share) {
    for (int o = 16; o >= 1; o >>= 1) tot.count += __shfl_xor_sync(kFull, tot.count, o);
    tot.dangling = __reduce_add_sync(kFull, tot.dangling);
    tot.qmax = __reduce_max_sync(kFull, tot.qmax);
    if ((threadIdx.x & 31) == 0) {
        if (tot.count) atomicAdd(&share.count, tot.count);
        if (tot.dangling) atomicAdd(&share.dangling, tot.dangling);
        if (tot.qmax) atomicMax(&share.qmax, tot.qmax);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (share.count) atomicAdd(&ctl->pcount[nslot], share.count);
        if (share.dangling) atomicAdd(&ctl->dctr[nslot], share.dangling);
        if (share.qmax > kPullMaxQ) atomicOr(&ctl->pcount[nslot], kPullsEnd);
        share = PullTotals{0ull, 0u, 0};
    }
}

// Pull rounds of a graph whose row lists are at most one step per warp, from round `cur` (2 or later)
// until one that is not a pull with a frontier (the caller's).  A small graph's round is a chain of loads: the
// counts, the warp's row record, its in-edges, their sources' residuals.  Here the record and
// the in-edges (in shared memory, in the list stages that only push rounds use) stay with the warp for all
// rounds, and the gathers go out before the round's counts are known.  A query at scale 14 (8 edges per
// vertex) 0.449 -> 0.331 ms, scale 10 0.444 -> 0.293, scale 15 (16 per vertex) 0.746 -> 0.622; what is left
// of a round's 5 us is the barrier, one gather and the apply's FP64.
// false: the grid barrier gave up.
__device__ __forceinline__ bool ppr_rounds_one_step(const PprParams& p, int& cur, int& iters, unsigned F1,
                                                    StageSmemD& sm, PullTotals& share, GridBarrier* bar,
                                                    unsigned long long& tph) {
    TraversalCtl* ctl = p.ctl;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const unsigned gwarp = (unsigned)wib * gridDim.x + blockIdx.x;  // the warp's step: over all SMs first
    const RowLists& R = p.rows;
    const auto edge = [&](int u) {  // 8 x 32 in-edges: 4 x 32 in xd0, 2 x 32 each in v0 and d0
        int2* const at = u < 4   ? reinterpret_cast<int2*>(sm.xd0[wib]) + 32 * u
                         : u < 6 ? reinterpret_cast<int2*>(sm.v0[wib]) + 32 * (u - 4)
                                 : reinterpret_cast<int2*>(sm.d0[wib]) + 32 * (u - 6);
        return at + lane;
    };
    const bool seg = gwarp < R.n[0];
    int L = 32;
    int4 rec = make_int4(0, 0, 0, 0);
    int2 sg = make_int2(0, 0);
    bool mine = false;
    if (seg) {
        rec = __ldg(R.rec + gwarp);
        sg = __ldg(R.seg + gwarp);
    } else if (gwarp < R.unit[kRowClasses]) {
        int c = 1;
        unsigned n = R.n[1], off = R.off[1], first = R.unit[1];
#pragma unroll
        for (int k = 2; k < kRowClasses; ++k)
            if (gwarp >= R.unit[k]) {
                c = k;
                n = R.n[k];
                off = R.off[k];
                first = R.unit[k];
            }
        const int logL = 6 - c;
        L = 1 << logL;
        const unsigned row = ((gwarp - first) << (5 - logL)) + (unsigned)(lane >> logL);
        if (row < n) rec = __ldg(R.rec + off + row);
        mine = row < n && (lane & (L - 1)) == 0;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kLaneEdges; ++u) {
        const int i = (lane & (L - 1)) + u * L;
        *edge(u) = i < rec.z ? __ldg(p.adj_r + rec.y + i) : make_int2(0, 0);
    }
    for (;;) {
        const int b = cur & 1, slot = cur % 3, nslot = (cur + 1) % 3, fslot = (cur + 2) % 3;
        const float2* qin = p.qf[b];
        float2 q[kLaneEdges];
        int wb[kLaneEdges];
#pragma unroll
        for (int u = 0; u < kLaneEdges; ++u) {
            const int2 e = *edge(u);
            wb[u] = e.y;
            q[u] = e.y > 0 ? __ldca(qin + e.x) : make_float2(0.f, 0.f);
        }
        float q0 = 0.f, pr0 = 0.f;
        double r0 = 0.0;
        if (mine || (seg && lane == 0)) {
            q0 = ldcg(reinterpret_cast<const float*>(qin + rec.x));
            r0 = ldcg(p.res + rec.x);
            pr0 = ldcg(p.pr + rec.x);
        }
        const unsigned long long c = ldcg(&ctl->pcount[slot]);
        const unsigned F = pull_frontier(c), T = (unsigned)c, D = ldcg(&ctl->dctr[slot]);
        if (F == 0 || T == 0 || iters >= p.max_iter || (c & kPullsEnd)) return true;  // grid-uniform
        ++iters;
        if (gtid == 0) {
            ctl->qctr[fslot] = 0ull;
            ctl->tilectr[fslot] = 0u;
            ctl->listctr[fslot] = 0u;
            ctl->dctr[fslot] = 0u;
            ctl->pcount[fslot] = 0ull;
            ctl->popped += F + D;
            ctl->relaxed += T;
            ctl->touched += (unsigned)p.V;
        }
        if (cur == 2)  // as in ppr_persistent
            for (unsigned j = gtid; j < F1; j += nthreads) {
                const int v = ldcg(p.q[1] + j).x;
                if (__ldg(p.row_r + v) == __ldg(p.row_r + v + 1)) p.qf[1][v] = make_float2(0.f, 0.f);
            }
        PullTotals tot{0ull, 0u, 0};
        PullSums s{0.f, 0.f};
#pragma unroll
        for (int u = 0; u < kLaneEdges; ++u) pull_add(q[u], wb[u], s);
        const double m = pull_reduce(s, L);
        if (mine) pull_apply(p, p.qf[b ^ 1], rec.x, rec.w, m, q0, r0, pr0, tot);
        if (seg && lane == 0) {
            if (c2g_dbits(m) != 0ull) atomicAdd(p.msg + rec.x, m);
            __threadfence();  // the sum is in msg before the segment arrives
            if (atomicAdd(p.arrived + sg.x, 1u) == (unsigned)sg.y - 1u) {
                __threadfence();  // the other segments' sums are seen
                const double all = ldcg(p.msg + rec.x);
                p.msg[rec.x] = 0.0;
                p.arrived[sg.x] = 0u;
                pull_apply(p, p.qf[b ^ 1], rec.x, rec.w, all, q0, r0, pr0, tot);
            }
        }
        pull_totals(ctl, nslot, tot, share);
        if (!grid_sync(bar, &ctl->flags, p.barrier_ns)) return false;
        phase_mark(ctl->phase_ns, tph, 2);
        ++cur;
    }
}

// The frontier list of a round whose frontier a pull counted: its vertices are popped (those without
// out-edges for good), with the FP64 residual that res still holds (qf only says who is in it: its pair is cut),
// and the other parity's qf is cleared for the round's apply.
__device__ __forceinline__ void ppr_list(const PprParams& p, int b, const FrontierOut& out, WarpStage& fst) {
    const int lane = threadIdx.x & 31;
    const unsigned gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned V = (unsigned)p.V;
    for (unsigned v0 = gwarp * 32; v0 < V; v0 += nwarps * 32) {
        const unsigned v = v0 + (unsigned)lane;
        double r = 0.0;
        int deg = 0;
        if (v < V) {
            const float2 q = ldcg(p.qf[b] + v);
            p.qf[b ^ 1][v] = make_float2(0.f, 0.f);
            if (q.x != 0.f) {
                r = ldcg(p.res + v);
                p.res[v] = 0.0;
                deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
                if (deg == 0) p.qf[b][v] = make_float2(0.f, 0.f);
            }
        }
        stage_push(fst, out, deg > 0, (int)v, deg, 0.f, (1.0 - (double)p.alpha) * r);
    }
    stage_flush(fst, out);
}

__global__ void __launch_bounds__(kPprThreads, kPprBlocksPerSm) ppr_persistent(const PprParams p) {
    TraversalCtl* ctl = p.ctl;
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(&ctl->bar_count);
    grid_sync_init();
    int* flags = &ctl->flags;
    const int lane = threadIdx.x & 31;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nthreads = gridDim.x * blockDim.x;
    const unsigned gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const unsigned V = (unsigned)p.V;
    const double a = (double)p.alpha, one_m_a = 1.0 - (double)p.alpha, absorb = (double)p.absorb;
    const unsigned long long rmax_bits = c2g_dbits((double)p.rmax);
    __shared__ StageSmemD sm;
    const int wib = threadIdx.x >> 5;
    WarpStage fst{sm.v0[wib], sm.d0[wib], nullptr, 0, sm.xd0[wib]};
    WarpStage tst{sm.v1[wib], nullptr, nullptr, 0};
    __shared__ PullTotals share;
    if (threadIdx.x == 0) share = PullTotals{0ull, 0u, 0};
    unsigned long long tph = globaltimer_ns();

    int sbase = p.st->stamp_base;
    const bool reset = sbase > (1 << 29);
    if (reset) sbase = 0;

    // Init: pr = res = msg = 0 (src/ppr/purn/Main.cu:156-169), qf = 0.
    for (unsigned v = gtid; v < V; v += nthreads) {
        p.pr[v] = 0.f;
        p.res[v] = 0.0;
        p.msg[v] = 0.0;
        p.qf[0][v] = p.qf[1][v] = make_float2(0.f, 0.f);
        if (reset) p.stamp[v] = -1;
    }
    if (!grid_sync(bar, flags, p.barrier_ns)) return;

    int qmax = 0;  // largest pushed residual this thread set outside a pull (float bits)
    const int s = p.source;
    const int s_deg = __ldg(p.row + s + 1) - __ldg(p.row + s);
    if (p.src_list) {
        // Several sources with their own residual (the adjoint's target set).
        const FrontierOut out = ppr_out(p, 1, 1);
        if (gtid == 0) ctl->seeds = p.n_src;
        for (unsigned b = gwarp * 32; b < (unsigned)p.n_src; b += nwarps * 32) {
            const unsigned i = b + (unsigned)lane;
            bool want = false, dang = false;
            int v = 0, deg = 0;
            double r = 0.0;
            if (i < (unsigned)p.n_src) {
                v = p.src_list[i];
                r = (double)p.src_r0[i];
                p.pr[v] = (float)(absorb * r);
                deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
                want = deg > 0;
                dang = !want;
                if (dang) p.res[v] = r;
                r *= one_m_a;
                p.qf[1][v] = ppr_pair(r);
            }
            stage_push(fst, out, want, v, deg, 0.f, r);
            list_push(p.dangle, &ctl->dctr[1], (unsigned)p.V, flags, dang, v);
        }
        stage_flush(fst, out);
    } else if (!p.seeded) {
        // Base init (src/ppr/base/Main.cu:146-150): residual r0 on the source, pr0 added
        // to pr[source]; the source is the round-1 frontier and is popped (res = 0).
        if (gwarp == 0) {
            if (lane == 0) {
                p.pr[s] = p.pr0;
                ctl->seeds = 0;
                p.qf[1][s] = ppr_pair(one_m_a * (double)p.r0);
                if (s_deg == 0) {
                    p.res[s] = (double)p.r0;
                    p.dangle[0] = s;
                    ctl->dctr[1] = 1;
                }
            }
            const FrontierOut out = ppr_out(p, 1, 1);
            stage_push(fst, out, lane == 0 && s_deg > 0, s, s_deg, 0.f, one_m_a * (double)p.r0);
            stage_flush(fst, out);
        }
    } else {
        // Pruned-graph init (src/ppr/purn/Main.cu:78-101,173-198): pr[s] = alpha; every
        // seed, i.e. the source's pruned records followed by its kept out-edges, adds
        // (1-alpha)*alpha*w to pr and (1-alpha)*w to res; all seeds form round 1.
        const unsigned n = (unsigned)p.n_rec + (unsigned)s_deg;
        if (gtid == 0) {
            atomicAdd(p.pr + s, p.alpha);
            ctl->seeds = n;
        }
        const int rs = __ldg(p.row + s);
        for (unsigned i = gtid; i < n; i += nthreads) {
            int v;
            float w;
            if (i < (unsigned)p.n_rec) {
                v = p.seed_v[i];
                w = p.seed_w[i];
            } else {
                const int2 ew = __ldg(p.adj + rs + (int)(i - (unsigned)p.n_rec));
                v = ew.x;
                w = __int_as_float(ew.y);
            }
            atomicAdd(p.pr + v, (float)(one_m_a * a * (double)w));
            atomicAdd(p.res + v, one_m_a * (double)w);
        }
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        const FrontierOut out = ppr_out(p, 1, 1);
        const int tag = sbase;  // distinct from every round's tag
        for (unsigned b = gwarp * 32; b < n; b += nwarps * 32) {
            const unsigned i = b + (unsigned)lane;
            bool want = false, dang = false;
            int v = 0, deg = 0;
            double r = 0.0;
            if (i < n) {
                v = (i < (unsigned)p.n_rec) ? p.seed_v[i] : __ldg(p.adj + rs + (int)(i - (unsigned)p.n_rec)).x;
                if (ldcg(p.stamp + v) != tag && atomicExch(p.stamp + v, tag) != tag) {
                    r = __ldcg(p.res + v);
                    deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
                    want = deg > 0;
                    dang = !want;
                    if (want) p.res[v] = 0.0;
                    r *= one_m_a;
                    const float2 q = ppr_pair(r);
                    p.qf[1][v] = q;
                    qmax = max(qmax, __float_as_int(q.x));  // a record's weight may be as large as a float
                }
            }
            stage_push(fst, out, want, v, deg, 0.f, r);
            list_push(p.dangle, &ctl->dctr[1], (unsigned)p.V, flags, dang, v);
        }
        if (qmax > kPullMaxQ) atomicMax(&ctl->farmin[1], qmax);
        stage_flush(fst, out);
    }
    if (!grid_sync(bar, flags, p.barrier_ns)) return;
    phase_mark(ctl->phase_ns, tph, 0);

    int cur = 1, iters = 0;
    unsigned F1 = 0;       // entries of round 1's list
    bool counted = false;  // this round's frontier is counted (a pull made it), not listed
    bool kept = false;     // ppr_rounds_one_step has run
    for (;;) {
        const int buf = cur & 1, slot = cur % 3, nslot = (cur + 1) % 3, fslot = (cur + 2) % 3;
        const unsigned long long c = counted ? ldcg(&ctl->pcount[slot]) : ldcg(&ctl->qctr[slot]);
        const unsigned F = pull_frontier(c), T = (unsigned)c;
        const unsigned D = ldcg(&ctl->dctr[slot]);
        if (F == 0 && D == 0) break;
        if (cur == 1) F1 = F;
        if (++iters > p.max_iter) {
            // Round cap (src/ppr/purn/Main.cu:224): the activated vertices keep their
            // residual, as in the reference where they are never popped (after a pull
            // res still holds it).
            if (gtid == 0) atomicOr(flags, C2G_FLAG_ITER_CAP);
            if (!counted)
                for (unsigned j = gtid; j < F; j += nthreads)
                    p.res[ldcg(p.q[buf] + j).x] = ldcg(p.qval[buf] + j) / one_m_a;
            break;
        }
        // grid-uniform; float pairs hold the pushed residuals and their sums below kPullMaxQ
        const bool large = counted ? (c & kPullsEnd) != 0 : ldcg(&ctl->farmin[slot]) != 0;
        const bool pull = T > (counted ? p.pull_next : p.pull_min) && !large;
        // Pop the activated vertices without out-edges: their residual is dropped.  A pull does so
        // for every vertex with in-edges.
        if (!counted) {
            for (unsigned j = gtid; j < D; j += nthreads) {
                const int v = ldcg(p.dangle + j);
                if (pull && __ldg(p.row_r + v) < __ldg(p.row_r + v + 1)) continue;
                p.res[v] = 0.0;
                p.qf[buf][v] = make_float2(0.f, 0.f);
            }
        } else if (F == 0) {
            for (unsigned v = gtid; v < V; v += nthreads)
                if (ldcg(p.qf[buf] + v).x != 0.f) p.res[v] = 0.0;
        }
        if (F == 0) {
            if (gtid == 0) ctl->popped += D;
            break;
        }
        if (gtid == 0) {
            ctl->qctr[fslot] = 0ull;
            ctl->tilectr[fslot] = 0u;
            ctl->listctr[fslot] = 0u;
            ctl->dctr[fslot] = 0u;
            ctl->pcount[fslot] = 0ull;
            ctl->farmin[fslot] = 0;
            if (large) atomicMax(&ctl->farmin[nslot], 1);
            ctl->popped += F + D;
            ctl->relaxed += T;
        }
        if (pull) {
            // Round 1's frontier may hold vertices without in-edges, which no pull visits: out of qf[1]
            // before round 3 reads it.
            if (cur == 2)
                for (unsigned j = gtid; j < F1; j += nthreads) {
                    const int v = ldcg(p.q[1] + j).x;
                    if (__ldg(p.row_r + v) == __ldg(p.row_r + v + 1)) p.qf[1][v] = make_float2(0.f, 0.f);
                }
            PullTotals tot{0ull, 0u};
            ppr_pull(p, buf, tot);
            pull_totals(ctl, nslot, tot, share);
            if (gtid == 0) ctl->touched += V;
            if (!grid_sync(bar, flags, p.barrier_ns)) return;
            phase_mark(ctl->phase_ns, tph, 2);
            counted = true;
            ++cur;
            if (p.one_step && !kept) {
                kept = true;
                if (!ppr_rounds_one_step(p, cur, iters, F1, sm, share, bar, tph)) return;
            }
            continue;
        }
        if (counted) {
            ppr_list(p, buf, ppr_out(p, buf, slot), fst);
            if (!grid_sync(bar, flags, p.barrier_ns)) return;
            phase_mark(ctl->phase_ns, tph, 1);
            counted = false;
        }
        const bool dense = p.dense_div > 0 && (unsigned long long)T * (unsigned)p.dense_div > p.E;
        const FrontierOut out = ppr_out(p, (cur + 1) & 1, nslot);
        ppr_push(p, buf, slot, F, T, tst, !dense);
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        phase_mark(ctl->phase_ns, tph, 2);
        if (!dense) {
            // Phase B: apply messages and activate (src/ppr/purn/Main.cu:383-391).
            const unsigned n = ldcg(&ctl->listctr[slot]);
            if (gtid == 0) ctl->touched += n;
            for (unsigned b = gwarp * 32; b < n; b += nwarps * 32) {
                const unsigned i = b + (unsigned)lane;
                bool want = false, dang = false;
                int v = 0, deg = 0;
                double r = 0.0;
                if (i < n) {
                    v = ldcg(p.touched + i);
                    r = __ldcg(p.res + v) + __ldcg(p.msg + v);
                    p.msg[v] = 0.0;
                    if (c2g_dbits(r) > rmax_bits) {  // both non-negative
                        p.pr[v] = ldcg(p.pr + v) + (float)(absorb * r);
                        deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
                        want = deg > 0;
                        dang = !want;
                        p.res[v] = want ? 0.0 : r;
                        r *= one_m_a;
                        const float2 q = ppr_pair(r);
                        p.qf[buf ^ 1][v] = q;
                        qmax = max(qmax, __float_as_int(q.x));
                    } else {
                        p.res[v] = r;
                    }
                }
                stage_push(fst, out, want, v, deg, 0.f, r);
                list_push(p.dangle, &ctl->dctr[nslot], (unsigned)p.V, flags, dang, v);
            }
        } else {
            // Dense apply: every vertex (an untouched one has msg 0 and res <= rmax, so
            // it is left as it is).
            if (gtid == 0) ctl->touched += V;
            for (unsigned b = gwarp * 32; b < V; b += nwarps * 32) {
                const unsigned v = b + (unsigned)lane;
                bool want = false, dang = false;
                int deg = 0;
                double r = 0.0;
                if (v < V) {
                    const double m = __ldcg(p.msg + v);
                    if (c2g_dbits(m) != 0ull) {  // messages are positive; msg is +0 otherwise
                        p.msg[v] = 0.0;
                        r = __ldcg(p.res + v) + m;
                        if (c2g_dbits(r) > rmax_bits) {  // both non-negative
                            p.pr[v] = ldcg(p.pr + v) + (float)(absorb * r);
                            deg = __ldg(p.row + v + 1) - __ldg(p.row + v);
                            want = deg > 0;
                            dang = !want;
                            p.res[v] = want ? 0.0 : r;
                            r *= one_m_a;
                            const float2 q = ppr_pair(r);
                            p.qf[buf ^ 1][v] = q;
                            qmax = max(qmax, __float_as_int(q.x));
                        } else {
                            p.res[v] = r;
                        }
                    }
                }
                stage_push(fst, out, want, (int)v, deg, 0.f, r);
                list_push(p.dangle, &ctl->dctr[nslot], (unsigned)p.V, flags, dang, (int)v);
            }
        }
        stage_flush(fst, out);
        if (qmax > kPullMaxQ) atomicMax(&ctl->farmin[nslot], qmax);
        if (!grid_sync(bar, flags, p.barrier_ns)) return;
        phase_mark(ctl->phase_ns, tph, 1);
        ++cur;
    }
    if (gtid == 0) {
        ctl->iterations = iters;
        p.st->stamp_base = sbase + cur + 2;
    }
}

__global__ void res_to_float(const double* __restrict__ r, float* __restrict__ out, int V) {
    const int stride = gridDim.x * blockDim.x;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += stride) out[v] = (float)r[v];
}

// Owner markers of a CSR: mark[t] = the largest v with row[v] <= t * 2^log_tile.
__global__ void csr_tile_markers(const int* __restrict__ row, int V, unsigned ntiles, int log_tile,
                                 int* __restrict__ mark) {
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) {
        const long long e = (long long)t << log_tile;
        int lo = 0, hi = V;
        while (hi - lo > 1) {
            const int mid = lo + ((hi - lo) >> 1);
            if ((long long)row[mid] <= e)
                lo = mid;
            else
                hi = mid;
        }
        mark[t] = lo;
    }
}

// ---------------------------------------------------------------------------------------
// host side

int build_markers(c2g_graph* g, const int* row, int** out) {
    const unsigned ntiles = (unsigned)(((size_t)g->E + (1u << kPullTileLog) - 1) >> kPullTileLog) + 1;
    C2G_CUDA(cudaMalloc(out, sizeof(int) * ntiles));
    csr_tile_markers<<<g->num_sms * 4, 256, 0, g->stream>>>(row, g->V, ntiles, kPullTileLog, *out);
    C2G_CUDA(cudaGetLastError());
    C2G_CUDA(cudaStreamSynchronize(g->stream));
    return C2G_OK;
}

static int ppr_geometry(c2g_graph* g) {
    if (g->geom_ppr.blocks > 0) return C2G_OK;
    int coop = 0;
    C2G_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g->device));
    if (!coop) return fail(C2G_ERR_UNSUPPORTED, "device %d lacks cooperative launch", g->device);
    int per_sm = 0;
    C2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ppr_persistent, kPprThreads, 0));
    if (per_sm < 1) return fail(C2G_ERR_CUDA, "PPR kernel cannot be resident (occupancy 0)");
    g->geom_ppr.blocks = per_sm * g->num_sms;
    g->geom_ppr.threads = kPprThreads;
    return C2G_OK;
}

void ppr_free(c2g_graph* g) {
    PprWork& w = g->ppr;
    void* ptrs[] = {w.pr, w.res, w.msg, w.qf[0], w.qf[1], w.arrived, w.res_f, w.stamp, w.q[0], w.q[1], w.qval[0], w.qval[1],
                    w.mark[0], w.mark[1], w.touched, w.dangle, w.ctl, w.st};
    for (void* ptr : ptrs)
        if (ptr) cudaFree(ptr);
    w = PprWork();
}

static int ppr_alloc(c2g_graph* g) {
    PprWork& w = g->ppr;
    const int log_tile = g->ppr_cfg.log_tile;
    if (w.msg && w.log_tile == log_tile) return C2G_OK;
    if (w.pr) ppr_free(g);
    const size_t nv = g->V ? (size_t)g->V : 1;
    const unsigned mark_cap = (unsigned)(((size_t)g->E >> log_tile) + 2);
    C2G_CUDA(cudaMalloc(&w.pr, sizeof(float) * nv));
    C2G_CUDA(cudaMalloc(&w.res, sizeof(double) * nv));
    C2G_CUDA(cudaMalloc(&w.msg, sizeof(double) * nv));
    C2G_CUDA(cudaMalloc(&w.res_f, sizeof(float) * nv));
    C2G_CUDA(cudaMalloc(&w.stamp, sizeof(int) * nv));
    C2G_CUDA(cudaMalloc(&w.touched, sizeof(int) * nv));
    C2G_CUDA(cudaMalloc(&w.dangle, sizeof(int) * nv));
    for (int b = 0; b < 2; ++b) {
        C2G_CUDA(cudaMalloc(&w.q[b], sizeof(int2) * nv));
        C2G_CUDA(cudaMalloc(&w.qval[b], sizeof(double) * nv));
        C2G_CUDA(cudaMalloc(&w.qf[b], sizeof(float2) * nv));
        C2G_CUDA(cudaMalloc(&w.mark[b], sizeof(int) * mark_cap));
    }
    C2G_CUDA(cudaMalloc(&w.ctl, sizeof(TraversalCtl)));
    C2G_CUDA(cudaMalloc(&w.st, sizeof(StampState)));
    C2G_CUDA(cudaMemsetAsync(w.stamp, 0xff, sizeof(int) * nv, g->stream));
    C2G_CUDA(cudaMemsetAsync(w.st, 0, sizeof(StampState), g->stream));
    w.mark_cap = mark_cap;
    w.log_tile = log_tile;
    return C2G_OK;
}

// Out-edges of the frontier above which a round pulls (~0: never).  A pull costs its pass over all
// in-edges, a push its frontier's out-edges (L2 atomics, 6.6e10 a second) and two barriers: at scale 20
// (16M edges) a pull takes 94 us, and a query 4.46 ms with pulls above E / 3, 4.49 above E / 2, 4.51
// above E / 5 and 6.05 with pulls only.  On small graphs a pull is about as short as the two
// barriers and dependent atomics of the emptiest push round: up to kPullAlwaysEdges every round pulls, and up to
// kPullMostEdges every round but those of a few thousand edges, which are all there is of a local query (large
// rmax); up to kPullTailEdges only those of at most E / kTailPullDiv before the first pull.  us a query, pulls above E / 3, E / 200, always:
// 1.2M edges (100,000 uniform vertices), rmax 1e-3 102 / 102 / 75, 1e-7 1273 / 1043 / 900; 2.1M (150,000) 90 /
// 90 / 80, 1358 / 1198 / 1132; 3.7M (scale 18) 110 / 106 / 124, 1770 / 1747 / 1798; 3.9M (299,999) 92 / 93 /
// 118, 1553 / 1460 / 1518; rmax 0.1 37 / 37 / 34, 32 / 32 / 36, 38 / 38 / 57, 38 / 38 / 58.
//
// Pulls sum float pairs, so they need
// weights below 2^30, a start below 2^60 and rmax of at least 1e-30 (as the batched push's pulls do),
// and alpha < 1: a residual of 0 pushed at alpha = 1 cannot be told from a vertex outside the
// frontier.
constexpr int64_t kPushPullDiv = 3;
constexpr int64_t kPullAlwaysEdges = 1600000, kPullTailEdges = 2500000, kPullMostEdges = 4000000;
constexpr int64_t kMostPullDiv = 200, kTailPullDiv = 1000;

static int ppr_pull_min(c2g_graph* g, const c2g_ppr_params& pp, const RowLists& rows, unsigned* pull_min,
                        unsigned* pull_next) {
    *pull_min = *pull_next = ~0u;
    const int div = g->ppr_cfg.pull_div;
    if (!rows.rec || !(pp.alpha < 1.f) || !(pp.rmax >= 1e-30f) || !(pp.r0 < 1e18f) || div == 0)
        return C2G_OK;
    int rc;
    if (!g->borrowed && (rc = ppr_pull_prepare(g))) return rc;
    if (!g->wstat_valid || g->wstat_wmax_bits >= kPullMaxWeight) return C2G_OK;
    if (div > 0) {
        *pull_min = *pull_next = (unsigned)(g->E / div);
        return C2G_OK;
    }
    const unsigned min = (unsigned)(g->E / (g->E <= kPullTailEdges   ? kTailPullDiv
                                            : g->E <= kPullMostEdges ? kMostPullDiv
                                                                     : kPushPullDiv));
    *pull_min = g->E <= kPullAlwaysEdges ? 0u : min;
    *pull_next = g->E <= kPullTailEdges ? 0u : min;
    return C2G_OK;
}

int ppr_launch_view(c2g_graph* g, const int32_t* row, const int2* adj, const int32_t* row_rev, const int2* adj_rev,
                    const RowLists& rows_rev, int32_t source, const c2g_ppr_params& pp, float absorb, int32_t n_src,
                    const int32_t* src_list, const float* src_r0, const int32_t* seed_v, const float* seed_w,
                    int32_t n_rec, float* pr_dev, float* res_dev, float* ms) {
    int rc;
    if ((rc = ppr_geometry(g))) return rc;
    if ((rc = ppr_alloc(g))) return rc;
    if (!adj) return fail(C2G_ERR_UNSUPPORTED, "graph has no float weights (flist / ppr wlist)");
    PprWork& w = g->ppr;
    PprParams p;
    p.row = row;
    p.adj = adj;
    p.V = g->V;
    p.E = (unsigned)g->E;
    p.row_r = row_rev;
    p.adj_r = adj_rev;
    p.rows = rows_rev;
    p.arrived = w.arrived;
    if ((rc = ppr_pull_min(g, pp, rows_rev, &p.pull_min, &p.pull_next))) return rc;
    p.one_step = false;
    p.dense_div = g->ppr_cfg.dense_div;
    p.pr = pr_dev ? pr_dev : w.pr;
    p.res = w.res;
    p.msg = w.msg;
    p.qf[0] = w.qf[0];
    p.qf[1] = w.qf[1];
    p.stamp = w.stamp;
    for (int b = 0; b < 2; ++b) {
        p.q[b] = w.q[b];
        p.qval[b] = w.qval[b];
        p.mark[b] = w.mark[b];
    }
    p.touched = w.touched;
    p.dangle = w.dangle;
    p.ctl = w.ctl;
    p.st = w.st;
    p.source = source;
    p.alpha = pp.alpha;
    p.rmax = pp.rmax;
    p.r0 = pp.r0;
    p.pr0 = pp.pr0;
    p.absorb = absorb;
    p.n_src = n_src;
    p.src_list = src_list;
    p.src_r0 = src_r0;
    p.max_iter = pp.max_iter;
    p.seeded = pp.seeded;
    p.seed_v = seed_v;
    p.seed_w = seed_w;
    p.n_rec = n_rec;
    p.log_tile = w.log_tile;
    p.mark_cap = w.mark_cap;
    p.barrier_ns = g->barrier_ns ? g->barrier_ns : 2000000000ull;
    int blocks = g->geom_ppr.blocks;
    if (p.pull_min != ~0u) {
        if (w.arrived_cap < rows_rev.n_long) {
            if (w.arrived) cudaFree(w.arrived);
            w.arrived = nullptr;
            w.arrived_cap = 0;
            C2G_CUDA(cudaMalloc(&w.arrived, sizeof(unsigned) * rows_rev.n_long));
            w.arrived_cap = rows_rev.n_long;
        }
        p.arrived = w.arrived;
        if (rows_rev.n_long)
            C2G_CUDA(cudaMemsetAsync(w.arrived, 0, sizeof(unsigned) * rows_rev.n_long, g->stream));
        // every round pulls: one warp per step of the row lists is enough, over all SMs (the applies of
        // an SM's warps share its FP64 pipe: scale 14 0.368 ms a query on 82 full blocks, 0.331 so)
        if (p.pull_min == 0u) {
            const unsigned units = rows_rev.unit[kRowClasses], warps = kPprThreads / 32;
            blocks = std::min(blocks, std::max((int)((units + warps - 1) / warps),
                                               std::min(g->num_sms, (int)((units + kStepsPerBlock - 1) / kStepsPerBlock))));
            p.one_step = units <= (unsigned)blocks * warps && rows_rev.segment <= 32 * kLaneEdges;
        }
    }
    C2G_CUDA(cudaMemsetAsync(w.ctl, 0, sizeof(TraversalCtl), g->stream));
    void* args[] = {&p};
    C2G_CUDA(cudaEventRecord(g->ev0, g->stream));
    C2G_CUDA(cudaLaunchCooperativeKernel((const void*)ppr_persistent, dim3(blocks),
                                         dim3(g->geom_ppr.threads), args, 0, g->stream));
    C2G_CUDA(cudaEventRecord(g->ev1, g->stream));
    // FP64 residuals reach the caller as float.
    res_to_float<<<g->num_sms * 4, 256, 0, g->stream>>>(w.res, res_dev ? res_dev : w.res_f, g->V);
    C2G_CUDA(cudaGetLastError());
    if (ms) {
        C2G_CUDA(cudaEventSynchronize(g->ev1));
        C2G_CUDA(cudaEventElapsedTime(ms, g->ev0, g->ev1));
    }
    return C2G_OK;
}

int ppr_launch(c2g_graph* g, int32_t source, const c2g_ppr_params& pp, const int32_t* seed_v,
               const float* seed_w, int32_t n_rec, float* pr_dev, float* res_dev, float* ms) {
    if (!g->adj_f) return fail(C2G_ERR_UNSUPPORTED, "graph has no float weights (flist)");
    int rc = C2G_OK;
    if (g->ppr_cfg.pull_div != 0) rc = g->ppr_cfg.pull_div > 0 ? build_reverse_graph(g) : ensure_reverse(g);
    if (rc) return rc;
    return ppr_launch_view(g, g->row, g->adj_f, g->row_r, g->adj_r, g->rows_in, source, pp, pp.alpha, 0, nullptr,
                           nullptr, seed_v, seed_w, n_rec, pr_dev, res_dev, ms);
}

}  // namespace c2g
