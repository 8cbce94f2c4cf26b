// Adsorption label propagation for sm_103a.
//
// The reference's "adsorption" programs are the PPR push with a different start
// (src/adsorption/w-base/Main.cu:124-395, served here by c2g_ppr with
// c2g_ppr_default_params(g, 1, ...)); they carry no labels.  This file is the
// label-propagation form of adsorption that the serving configuration asks for:
//     Y_v <- p_inj(v) * I_v + p_cont(v) * sum_{u->v} w(u,v) * Y_u
// over L = 16 labels per query (I_v = 1 for the vertex seeding label l), iterated a
// fixed number of times from Y = I.  The abandonment share p_abnd(v) goes to the dummy
// "none" label, which is not stored.
//
// One iteration is one kernel: a pull over the reverse CSR that applies p_inj / p_cont on
// the spot and writes the next label rows, between two row buffers.  The in-edges of all
// vertices form one range [0, E) cut into tiles, one per warp, and a tile into eight equal
// stretches, one per group of 4 lanes (each lane holds 4 of the 16 labels).  A group walks
// its stretch in order: the in-edges come through shared memory 32 (small graphs: 8) at a
// time (cp.async, two buffers), the label rows of kAdsBatch in-edges are in flight while those
// before them are summed, and a bitmap of row starts says where a row ends.  A row that lies inside a
// stretch is written by its group; one that crosses stretches is summed over the groups by
// shuffles; one that crosses tiles leaves a partial sum per tile, and the warp that arrives
// last adds them up, in order.
// What bounds a large graph is the label-row gathers, 64 bytes per in-edge: 65 M of them
// take 0.55 ms an iteration at scale 22, 7.6 TB/s into the SMs (a third of the rows from
// DRAM).  Before, a group found each row's end in the row pointer (a dependent load per
// row), wrote sums to memory for a vertex pass, and an iteration took 1.40 ms.  30 iterations
// at scale 22: 16.1 ms with 2 rows ahead and 8 blocks per SM (16.6 while it spilled, as the others did); 17.0 with 7; 18.0 with 4 rows
// ahead and 8 blocks, 17.8 with 6, 21.5 with 8 rows and 4 blocks: more warps, each with fewer
// rows in registers.  What bounds a small one is the chain of loads through a stretch.
// Per iteration: (8 + 64) bytes per edge (in-edge record + source label row) and
// 64 + 16 bytes per vertex with in-edges.  The iteration sequence is captured once per
// handle (and iteration count) into a CUDA graph and replayed; its buffers stay with the
// handle.
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

namespace c2g {

constexpr int kAdsL = 16;          // labels per query

constexpr int kAdsBatch = 2;       // in-edges whose label rows a group gathers ahead
constexpr int kAdsMinBlocks = 8;   // launch bounds: resident 128-thread blocks per SM
constexpr int kAdsThreads = 128;
constexpr int kAdsWarps = kAdsThreads / 32;
constexpr unsigned kAdsBareBlocks = 64;  // blocks that write the listed rows without in-edges

struct AdsPass {
    const int* row_r;
    const int2* adj_r;
    const unsigned* r_bits;   // per chunk of 32 in-edges: which start a row,
    const int* r_prefix;      // and how many rows start in earlier chunks
    const int4* coef;         // per row with in-edges, in order: vertex, p_cont, p_inj, seed mask; from the
    const unsigned* n_bare;   // end, this many rows without in-edges whose labels are not 0 after an iteration
    const float* p_inj;
    float4* slots;            // per tile: sum of the row that enters it, of the row that leaves it
    unsigned* arrived;        // per tile: tiles of the row leaving it that have left their sums
    int V;
    unsigned E;
    int tile_log;             // a tile holds 2^tile_log in-edges, eight stretches of whole chunks
};

__device__ __forceinline__ void ads_apply(float4* __restrict__ out, const int4 c, int part, const float4 s) {
    const float pc = __int_as_float(c.y), pi = __int_as_float(c.z);
    const int m = c.w >> (4 * part);
    float4 y;
    y.x = fmaf(pc, s.x, m & 1 ? pi : 0.f);
    y.y = fmaf(pc, s.y, m & 2 ? pi : 0.f);
    y.z = fmaf(pc, s.z, m & 4 ? pi : 0.f);
    y.w = fmaf(pc, s.w, m & 8 ? pi : 0.f);
    out[(size_t)c.x * (kAdsL / 4) + part] = y;
}

__device__ __forceinline__ float4 ads_add(const float4 a, const float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

__device__ __forceinline__ float4 ads_shfl_up(const float4 a, int d) {
    return make_float4(__shfl_up_sync(~0u, a.x, d), __shfl_up_sync(~0u, a.y, d), __shfl_up_sync(~0u, a.z, d),
                       __shfl_up_sync(~0u, a.w, d));
}

// out = p_cont * (sum over in-edges of w * Y) + p_inj * I for every vertex with in-edges; row V of Y is zero.
// C: in-edges a group stages in shared memory at a time.
template <int C>
__global__ void __launch_bounds__(kAdsThreads, kAdsMinBlocks)
    ads_iterate(const AdsPass p, const float4* __restrict__ Y, float4* __restrict__ out) {
    // each group's staged in-edges, two chunks; 16 bytes of padding per row, so that the 8
    // groups of a warp, reading 16 bytes of their rows at once, hit different banks
    __shared__ __align__(16) int2 staged[kAdsWarps][2][8][C + 2];
    __shared__ float4 heads[kAdsThreads];
    if (blockIdx.x < kAdsBareBlocks) {
        const unsigned n = 4u * __ldg(p.n_bare), step = min(gridDim.x, kAdsBareBlocks) * kAdsThreads;
        for (unsigned i = blockIdx.x * kAdsThreads + threadIdx.x; i < n; i += step)
            ads_apply(out, __ldg(p.coef + (p.V - 1 - (int)(i >> 2))), (int)(i & 3u), make_float4(0.f, 0.f, 0.f, 0.f));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int part = lane & 3, grp = lane >> 2;  // labels 4*part .. 4*part+3 of the group's rows
    const unsigned t = blockIdx.x * kAdsWarps + warp;
    const unsigned stretch = 1u << (p.tile_log - 3);
    const unsigned e0 = (t << p.tile_log) + (unsigned)grp * stretch;
    if ((t << p.tile_log) >= p.E) return;  // warp-uniform, no block barrier below
    const unsigned e1 = min(e0 + stretch, p.E);
    const bool act = e0 < p.E;
    const auto start_bits = [&](unsigned e) { return __ldg(p.r_bits + (e >> 5)) >> (e & 31u) & (~0u >> (32 - C)); };
    unsigned bits = act ? start_bits(e0) : 0u;
    const bool starts = bits & 1u;         // the stretch's first in-edge starts a row
    int first = 0;                         // its row
    if (act) {
        const unsigned before = C < 32 ? __ldg(p.r_bits + (e0 >> 5)) & ((1u << (e0 & 31u)) - 1u) : 0u;
        first = __ldg(p.r_prefix + (e0 >> 5)) + __popc(before) + (int)starts - 1;
    }
    int row = first;
    int4 coef = act ? __ldg(p.coef + first) : make_int4(0, 0, 0, 0);
    bits &= ~1u;
    bool head = !starts;                   // the row being summed began before the stretch
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);

    const auto stage = [&](unsigned c) {
        int2* const to = staged[warp][c & 1u][grp];
        const unsigned base = e0 + c * C;
        if (base + C <= p.E) {
#pragma unroll
            for (int r = 0; r < C / 8; ++r)
                cp_async16(to + 2 * part + 8 * r, p.adj_r + base + 2 * part + 8 * r);
        } else {  // beyond the last in-edge: the zero row
#pragma unroll 1
            for (unsigned i = part; i < C; i += 4)
                to[i] = base + i < p.E ? __ldg(p.adj_r + base + i) : make_int2(p.V, 0);
        }
    };
    float4 y[2][kAdsBatch];
    float w[2][kAdsBatch];
    const auto gather = [&](int b, const int2* from) {
#pragma unroll
        for (int k = 0; k < kAdsBatch; k += 2) {
            const int4 two = *reinterpret_cast<const int4*>(from + k);
            w[b][k] = __int_as_float(two.y);
            w[b][k + 1] = __int_as_float(two.w);
            y[b][k] = __ldg(Y + (size_t)two.x * (kAdsL / 4) + part);
            y[b][k + 1] = __ldg(Y + (size_t)two.z * (kAdsL / 4) + part);
        }
    };
    const auto consume = [&](int b) {
#pragma unroll
        for (int k = 0; k < kAdsBatch; ++k) {
            if (bits & (1u << k)) {  // a new row: the one before is complete
                if (head) {
                    heads[threadIdx.x] = s;
                    head = false;
                } else {
                    ads_apply(out, coef, part, s);
                }
                s = make_float4(0.f, 0.f, 0.f, 0.f);
                ++row;
                coef = __ldg(p.coef + row);
            }
            s.x = fmaf(w[b][k], y[b][k].x, s.x);
            s.y = fmaf(w[b][k], y[b][k].y, s.y);
            s.z = fmaf(w[b][k], y[b][k].z, s.z);
            s.w = fmaf(w[b][k], y[b][k].w, s.w);
        }
        bits >>= kAdsBatch;
    };

    const unsigned chunks = stretch / C;
    stage(0);
    cp_async_commit();
    if (chunks > 1) stage(1);
    cp_async_commit();
    cp_async_wait_but<1>();
    __syncwarp();
    gather(0, staged[warp][0][grp]);
    for (unsigned c = 0; c < chunks; ++c) {
        const int2* const st = staged[warp][c & 1u][grp];
        const unsigned next = e0 + (c + 1) * C;
        const unsigned next_bits = c + 1 < chunks && next < p.E ? start_bits(next) : 0u;
#pragma unroll 1
        for (int b = 0; b < C - 2 * kAdsBatch; b += 2 * kAdsBatch) {
            gather(1, st + b + kAdsBatch);
            consume(0);
            gather(0, st + b + 2 * kAdsBatch);
            consume(1);
        }
        gather(1, st + C - kAdsBatch);
        consume(0);
        if (c + 1 < chunks) {
            cp_async_wait_but<0>();
            __syncwarp();  // the next chunk is there, and this one is read
            if (c + 2 < chunks) stage(c + 2);
            cp_async_commit();
            gather(0, staged[warp][(c + 1) & 1u][grp]);
        }
        consume(1);
        bits = next_bits;
    }
    __syncwarp();

    // the row at the end of each stretch, summed over the stretches that it crosses
    const bool had_head = !starts && !head;  // a row that began before the stretch ended in it
    const bool done = act && (e1 == p.E || (start_bits(e1) & 1u));
    int f = starts || had_head;              // it began in the tile
#pragma unroll
    for (int d = 1; d < 8; d *= 2) {
        const float4 ps = ads_shfl_up(s, 4 * d);
        const int pf = __shfl_up_sync(~0u, f, 4 * d);
        if (grp >= d) {
            if (!f) s = ads_add(s, ps);
            f |= pf;
        }
    }
    float4 enter = ads_shfl_up(s, 4);
    int enter_f = __shfl_up_sync(~0u, f, 4);
    if (grp == 0) {
        enter = make_float4(0.f, 0.f, 0.f, 0.f);
        enter_f = 0;
    }
    if (had_head) {
        enter = ads_add(enter, heads[threadIdx.x]);
        if (enter_f) ads_apply(out, __ldg(p.coef + first), part, enter);
    }
    if (done && f) ads_apply(out, coef, part, s);
    // rows that cross tiles: at most one enters the tile (its group: in), one leaves it (out)
    const bool in_row = act && ((had_head && !enter_f) || (!f && (done || grp == 7)));
    const bool out_row = act && grp == 7 && !done && f;
    const unsigned any_in = __ballot_sync(~0u, in_row), any_out = __ballot_sync(~0u, out_row);
    if (!(any_in | any_out)) return;
    if (in_row) p.slots[(size_t)t * 8 + part] = had_head ? enter : s;
    if (out_row) p.slots[(size_t)t * 8 + 4 + part] = s;
    __threadfence();
    __syncwarp();
    unsigned ts[2] = {0, 0}, te[2] = {0, 0};
    int rows[2] = {0, 0};
    int last[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const unsigned any = k ? any_out : any_in;
        if (!any) continue;  // warp-uniform
        const int src = __ffs(any) - 1;
        rows[k] = __shfl_sync(~0u, k ? row : first, src);
        const int v = __ldg(&p.coef[rows[k]].x);
        ts[k] = (unsigned)__ldg(p.row_r + v) >> p.tile_log;
        te[k] = (unsigned)(__ldg(p.row_r + v + 1) - 1) >> p.tile_log;
        if (lane == 0) {
            last[k] = atomicAdd(p.arrived + ts[k], 1u) == te[k] - ts[k];
            if (last[k]) p.arrived[ts[k]] = 0u;  // for the next iteration
        }
    }
    __threadfence();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!__shfl_sync(~0u, last[k], 0)) continue;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        if (grp == 0) sum = __ldcg(p.slots + (size_t)ts[k] * 8 + 4 + part);
#pragma unroll 4
        for (unsigned i = ts[k] + 1 + (unsigned)grp; i <= te[k]; i += 8)
            sum = ads_add(sum, __ldcg(p.slots + (size_t)i * 8 + part));
#pragma unroll
        for (int d = 4; d < 32; d *= 2) {
            sum.x += __shfl_xor_sync(~0u, sum.x, d);
            sum.y += __shfl_xor_sync(~0u, sum.y, d);
            sum.z += __shfl_xor_sync(~0u, sum.z, d);
            sum.w += __shfl_xor_sync(~0u, sum.w, d);
        }
        if (grp == 0) ads_apply(out, __ldg(p.coef + rows[k]), part, sum);
    }
}

// Y0 = I (seed labels) and its zero row, Y1 = 0 for the rows that no iteration writes, and the coefficients of the
// rows with in-edges, in their order.  Of those without, the ones that an iteration leaves with other labels than 0
// are listed from coef's end: the seeds, which keep their injection alone, and those whose p_cont is not finite (it
// times an empty sum is NaN).
__global__ void ads_init(const AdsPass p, const float* __restrict__ p_cont, const unsigned* __restrict__ seedmask,
                         float4* __restrict__ Y0, float4* __restrict__ Y1, int4* __restrict__ coef,
                         unsigned* __restrict__ n_bare) {
    const size_t n = ((size_t)p.V + 1) * (kAdsL / 4);
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int v = (int)(i / (kAdsL / 4)), part = (int)(i % (kAdsL / 4));
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (v == p.V) {
            Y0[i] = zero;
            Y1[i] = zero;
            continue;
        }
        const unsigned mask = seedmask[v], m = mask >> (4 * part);
        Y0[i] = make_float4(m & 1u, (m >> 1) & 1u, (m >> 2) & 1u, (m >> 3) & 1u);
        const int r0 = __ldg(p.row_r + v);
        const bool bare = r0 == __ldg(p.row_r + v + 1);
        if (bare) Y1[i] = zero;
        if (part == 0) {
            const float pc = p_cont[v];
            const int4 c = make_int4(v, __float_as_int(pc), __float_as_int(p.p_inj[v]), (int)mask);
            if (!bare) {
                const unsigned before = __ldg(p.r_bits + (r0 >> 5)) & ((1u << (r0 & 31)) - 1u);
                coef[__ldg(p.r_prefix + (r0 >> 5)) + __popc(before)] = c;
            } else if (mask != 0u || !isfinite(pc)) {
                coef[p.V - 1 - (int)atomicAdd(n_bare, 1u)] = c;
            }
        }
    }
}

// Seed mask from the 16 seed vertices: bit l of mask[v] says label l is seeded at v.
__global__ void ads_seed_mask(const int* __restrict__ seeds, int n, unsigned* __restrict__ mask, unsigned* n_bare) {
    const int l = threadIdx.x;
    if (l == 0) *n_bare = 0u;
    if (l < n) atomicOr(mask + seeds[l], 1u << l);
}

// Per-handle workspace of the label propagation, kept across calls so that a serving
// loop's adsorption requests allocate nothing after the first one (cudaMalloc and
// cudaFree synchronise the device and would stall the other kinds' batches), with the
// iteration sequence captured once into a CUDA graph and replayed.
struct AdsWork {
    float* Y[2] = {nullptr, nullptr};  // [V + 1][16], row V zero
    int4* coef = nullptr;              // [V]
    float4* slots = nullptr;           // [tiles][2][16 floats]
    unsigned* arrived = nullptr;       // [tiles], zero between iterations
    unsigned* mask = nullptr;
    float* pi = nullptr;
    float* pc = nullptr;
    int* seeds = nullptr;  // [16], and the number of listed rows without in-edges behind them
    cudaGraphExec_t exec = nullptr;
    int iterations = -1;
    int tile_log = 0;
};

void ads_free(c2g_graph* g) {
    AdsWork* w = reinterpret_cast<AdsWork*>(g->ads);
    if (!w) return;
    if (w->exec) cudaGraphExecDestroy(w->exec);
    void* ptrs[] = {w->Y[0], w->Y[1], w->coef, w->slots, w->arrived, w->mask, w->pi, w->pc, w->seeds};
    for (void* q : ptrs)
        if (q) cudaFree(q);
    delete w;
    g->ads = nullptr;
}

// In-edges per tile (log2): eight stretches of 128, shorter ones where that leaves the SMs short of
// warps.  30 iterations at scale 22: 16.6 ms with 1024-edge tiles, 20.4 with 512, 25.8 with 256 (a
// tile's start and end are chains of loads); at scale 18 1.25 ms with 512, 1.36 with 256.  64-edge
// tiles, staged 8 in-edges at a time, where all of them are resident at once: there the walk along a
// stretch is what an iteration takes (scale 10 0.34 -> 0.20 ms, scale 14 0.40 -> 0.26, against 256; scale 15
// 0.42 either way, scale 16 0.48 -> 0.69).
static int ads_tile_log(const c2g_graph* g) {
    const int64_t warps = (int64_t)g->num_sms * kAdsMinBlocks * kAdsWarps;
    int log = 10;
    while (log > 8 && ((int64_t)g->E >> log) < warps) --log;
    if (((int64_t)g->E >> 6) < warps) log = 6;
    return log;
}

static int ads_alloc(c2g_graph* g, AdsWork** out) {
    AdsWork* w = reinterpret_cast<AdsWork*>(g->ads);
    if (!w) {
        w = new AdsWork();
        g->ads = w;
        const size_t V = g->V ? (size_t)g->V : 1;
        w->tile_log = ads_tile_log(g);
        const size_t tiles = ((size_t)g->E >> w->tile_log) + 1;
        cudaError_t e = cudaMalloc(&w->Y[0], sizeof(float) * (V + 1) * kAdsL);
        if (e == cudaSuccess) e = cudaMalloc(&w->Y[1], sizeof(float) * (V + 1) * kAdsL);
        if (e == cudaSuccess) e = cudaMalloc(&w->coef, sizeof(int4) * V);
        if (e == cudaSuccess) e = cudaMalloc(&w->slots, sizeof(float) * tiles * 2 * kAdsL);
        if (e == cudaSuccess) e = cudaMalloc(&w->arrived, sizeof(unsigned) * tiles);
        if (e == cudaSuccess) e = cudaMemsetAsync(w->arrived, 0, sizeof(unsigned) * tiles, g->stream);
        if (e == cudaSuccess) e = cudaMalloc(&w->mask, sizeof(unsigned) * V);
        if (e == cudaSuccess) e = cudaMalloc(&w->pi, sizeof(float) * V);
        if (e == cudaSuccess) e = cudaMalloc(&w->pc, sizeof(float) * V);
        if (e == cudaSuccess) e = cudaMalloc(&w->seeds, sizeof(int) * (kAdsL + 1));
        if (e != cudaSuccess) ads_free(g);
        C2G_CUDA(e);
    }
    *out = w;
    return C2G_OK;
}

// Capture init + `iterations` passes on the handle's stream; the result is in Y[iterations & 1].
static int ads_capture(c2g_graph* g, AdsWork* w, int iterations) {
    if (w->exec && w->iterations == iterations) return C2G_OK;
    if (w->exec) {
        cudaGraphExecDestroy(w->exec);
        w->exec = nullptr;
    }
    unsigned* const n_bare = reinterpret_cast<unsigned*>(w->seeds) + kAdsL;
    const AdsPass p{g->row_r, g->adj_r, g->r_bits, g->r_prefix, w->coef, n_bare, w->pi, w->slots, w->arrived,
                    g->V,     (unsigned)g->E, w->tile_log};
    const unsigned tile_edges = kAdsWarps << w->tile_log;
    const int blocks = (int)(((size_t)g->E + tile_edges - 1) / tile_edges);
    float4* const Y[2] = {reinterpret_cast<float4*>(w->Y[0]), reinterpret_cast<float4*>(w->Y[1])};
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(g->stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        ads_init<<<g->num_sms * 8, 256, 0, g->stream>>>(p, w->pc, w->mask, Y[0], Y[1], w->coef, n_bare);
        for (int it = 0; it < iterations; ++it)  // without in-edges one block writes the listed rows
            (w->tile_log < 8 ? ads_iterate<8> : ads_iterate<32>)<<<blocks ? blocks : 1, kAdsThreads, 0, g->stream>>>(p, Y[it & 1], Y[(it + 1) & 1]);
        e = cudaStreamEndCapture(g->stream, &graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&w->exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    C2G_CUDA(e);
    w->iterations = iterations;
    return C2G_OK;
}

}  // namespace c2g

using namespace c2g;

extern "C" int c2g_adsorption(c2g_graph* g, int32_t n_labels, const int32_t* seed_vertices, const float* p_inj,
                              const float* p_cont, const float* p_abnd, int32_t iterations, float* Y_out,
                              int on_device, c2g_stats* stats) {
    if (!g || !seed_vertices || !p_inj || !p_cont || !Y_out) return fail(C2G_ERR_ARG, "NULL argument");
    if (n_labels != kAdsL) return fail(C2G_ERR_UNSUPPORTED, "adsorption supports %d labels per query", kAdsL);
    if (iterations < 0) return fail(C2G_ERR_ARG, "iterations must be >= 0");
    if (!g->adj_f) return fail(C2G_ERR_UNSUPPORTED, "graph has no float weights (flist)");
    (void)p_abnd;  // the abandonment share goes to the unstored dummy label
    for (int32_t l = 0; l < n_labels; ++l)
        if (seed_vertices[l] < 0 || seed_vertices[l] >= g->V)
            return fail(C2G_ERR_RANGE, "seed vertex %d out of range", seed_vertices[l]);
    std::lock_guard<std::mutex> lk(g->mu);
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    struct Restore {
        int d;
        ~Restore() {
            if (d >= 0) cudaSetDevice(d);
        }
    } restore{prev};
    AdsWork* w = nullptr;
    int rc = with_room_of_rows(g, [&] {
        const int r = build_reverse_graph(g);
        return r ? r : ads_alloc(g, &w);
    });
    if (rc) return rc;
    const size_t V = (size_t)g->V;
    const cudaMemcpyKind in_kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    float ms = 0.f;
    cudaError_t e = cudaMemcpyAsync(w->seeds, seed_vertices, sizeof(int) * kAdsL, cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(w->pi, p_inj, sizeof(float) * V, in_kind, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(w->pc, p_cont, sizeof(float) * V, in_kind, g->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(w->mask, 0, sizeof(unsigned) * V, g->stream);
    if (e == cudaSuccess) {
        ads_seed_mask<<<1, 32, 0, g->stream>>>(w->seeds, kAdsL, w->mask, reinterpret_cast<unsigned*>(w->seeds) + kAdsL);
        e = cudaGetLastError();
    }
    C2G_CUDA(e);
    if ((rc = ads_capture(g, w, iterations))) return rc;
    e = cudaEventRecord(g->ev0, g->stream);
    if (e == cudaSuccess) e = cudaGraphLaunch(w->exec, g->stream);
    if (e == cudaSuccess) e = cudaEventRecord(g->ev1, g->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(Y_out, w->Y[iterations & 1], sizeof(float) * V * kAdsL,
                            on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    C2G_CUDA(e);
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->source = seed_vertices[0];
        stats->iterations = iterations;
        stats->edges_relaxed = (int64_t)g->E * iterations;
        stats->vertices_popped = (int64_t)g->V * iterations;
        stats->n_seeds = n_labels;
        stats->device_ms = ms;
        stats->alg_bytes = ((8.0 + 64.0) * (double)g->E + (64.0 + 16.0) * (double)g->V) * iterations;
    }
    return C2G_OK;
}
