// In-edge rows of a graph with int32 weights, ordered by weight: the layout of the SSSP
// pull rounds (sssp.cu, batch.cu).
//
// Row v holds v's in-edges (source, weight) in ascending order of weight, padded with
// (0, INT_MAX) to a multiple of 4 edges, so that a row is read in aligned 32-byte groups and
// a reader can stop at the first group whose weights cannot improve v any more.  The
// reference has no in-edges; it relaxes out-edges only (src/sssp/purn/Main.cu:236-331).
//
// Built on the device when the graph is made (its int32 weights never change): count the
// in-edges, scan the padded row lengths, scatter the edges into their rows, order each row.
// Rows of up to 32 edges are ordered by a warp (bitonic network on weight and source), longer
// ones by a block (counting sort over kInBuckets buckets of weight).  A bucket spans 2^shift
// weights, where 2^shift * kInBuckets covers the largest weight; inside a bucket the order is
// free, so a reader compares with the bucket's lower end, (w >> shift) << shift.  Each step is
// bound by scattered 8-byte accesses: at scale 22 (65M edges) making the graph from host
// arrays takes 68.2 ms with the rows and 63.5 ms without.
#include <climits>

#include "device_common.cuh"
#include "internal.h"

namespace c2g {
namespace {

constexpr int kInBuckets = 1024;
constexpr int kInSortThreads = 256;
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;  // rows per thread of a scan block

struct InStats {
    int wmin, wmax;
    unsigned n_long;             // rows longer than a warp
    unsigned n_seg;              // segments of rows longer than kInHead
    unsigned long long padded;   // padded edges of all rows
};

__global__ void in_count(const int2* __restrict__ adj, unsigned E, int* __restrict__ indeg, InStats* st) {
    const unsigned stride = gridDim.x * blockDim.x;
    int lo = INT_MAX, hi = INT_MIN;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
        const int2 ew = __ldg(adj + e);
        atomicAdd(indeg + ew.x, 1);
        lo = min(lo, ew.y);
        hi = max(hi, ew.y);
    }
    lo = __reduce_min_sync(kFull, lo);
    hi = __reduce_max_sync(kFull, hi);
    if ((threadIdx.x & 31) == 0) {
        if (lo < ldcg(&st->wmin)) atomicMin(&st->wmin, lo);
        if (hi > ldcg(&st->wmax)) atomicMax(&st->wmax, hi);
    }
}

__device__ __forceinline__ int padded4(int n) { return (n + 3) & ~3; }

// Exclusive sum over the block of one int per thread; *total (all threads) gets the block's sum.
__device__ __forceinline__ int block_exclusive(int x, int* total) {
    __shared__ int s_warp[kScanThreads / 32];
    __shared__ int s_total;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[wib] = incl;
    __syncthreads();
    if (wib == 0) {
        const int n = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
        int s = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, s, o);
            if (lane >= o) s += t;
        }
        if (lane < (int)(blockDim.x >> 5)) s_warp[lane] = s - n;
        if (lane == 31) s_total = s;
    }
    __syncthreads();
    *total = s_total;
    const int r = s_warp[wib] + incl - x;
    __syncthreads();
    return r;
}

// Padded edges of each scan block's rows (their sum may pass 2^31: st->padded).
__global__ void __launch_bounds__(kScanThreads) in_scan_blocks(const int* __restrict__ indeg, int V,
                                                              int* __restrict__ block_sum, InStats* st) {
    const int base = (int)blockIdx.x * kScanThreads * kScanItems;
    int n = 0;
    for (int k = 0; k < kScanItems; ++k) {
        const int v = base + k * kScanThreads + (int)threadIdx.x;
        if (v < V) n += padded4(__ldg(indeg + v));
    }
    int total;
    block_exclusive(n, &total);
    if (threadIdx.x == 0) {
        block_sum[blockIdx.x] = total;
        atomicAdd(&st->padded, (unsigned long long)total);
    }
}

// Exclusive sums of the scan blocks' totals, by one block.
__global__ void __launch_bounds__(kScanThreads) in_scan_sums(int* __restrict__ block_sum, int n) {
    int carry = 0;
    for (int b = 0; b < n; b += kScanThreads) {
        const int i = b + (int)threadIdx.x;
        const int x = i < n ? block_sum[i] : 0;
        int total;
        const int ex = block_exclusive(x, &total);
        if (i < n) block_sum[i] = carry + ex;
        carry += total;
    }
}

// Row starts, the scatter's cursors and the list of rows longer than a warp.
__global__ void __launch_bounds__(kScanThreads) in_scan_rows(const int* __restrict__ indeg, int V,
                                                            const int* __restrict__ block_sum, int* __restrict__ row,
                                                            int* __restrict__ cursor, int* __restrict__ longs,
                                                            InStats* st) {
    const int base = ((int)blockIdx.x * kScanThreads + (int)threadIdx.x) * kScanItems;
    int d[kScanItems], n = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        d[k] = base + k < V ? __ldg(indeg + base + k) : 0;
        n += padded4(d[k]);
    }
    int total;
    int at = block_sum[blockIdx.x] + block_exclusive(n, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int v = base + k;
        const bool lng = v < V && d[k] > 32;
        if (v < V && padded4(d[k]) > kInHead)
            atomicAdd(&st->n_seg, (unsigned)(padded4(d[k]) - kInHead + kInSegment - 1) / kInSegment);
        if (v < V) {
            row[v] = at;
            cursor[v] = at;
        }
        at += padded4(d[k]);
        if (v == V - 1) row[V] = at;
        list_push(longs, &st->n_long, (unsigned)V, reinterpret_cast<int*>(&st->n_long), lng, v);
    }
}

// The parts of long rows behind their first kInHead edges, kInSegment edges each: (vertex, first edge).
__global__ void in_segments(const int* __restrict__ row, const int* __restrict__ longs, unsigned n_long,
                            unsigned* __restrict__ ctr, unsigned n_seg, int2* __restrict__ seg) {
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned r = blockIdx.x * blockDim.x + threadIdx.x; r < n_long; r += stride) {
        const int v = __ldg(longs + r), re = __ldg(row + v + 1);
        const int first = __ldg(row + v) + kInHead;
        if (first >= re) continue;
        unsigned at = atomicAdd(ctr, (unsigned)(re - first + kInSegment - 1) / kInSegment);
        for (int i = first; i < re && at < n_seg; i += kInSegment) seg[at++] = make_int2(v, i);
    }
}

// Every out-edge u -> v into v's row, in any order.  A warp takes kScatterTile edges at a time
// whatever rows they belong to (a row may hold 100,000), finds the first one's row by
// bisection and loads 32 row starts at once from there on.
constexpr unsigned kScatterTile = 1024;

__global__ void in_scatter(const int* __restrict__ row, const int2* __restrict__ adj, int V, unsigned E,
                           int* __restrict__ cursor, int2* __restrict__ raw) {
    const int lane = threadIdx.x & 31;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned ntiles = (E + kScatterTile - 1) / kScatterTile;
    for (unsigned t = warp; t < ntiles; t += nwarps) {
        unsigned e0 = t * kScatterTile;
        const unsigned e1 = min(e0 + kScatterTile, E);
        int lo = 0, hi = V;  // row[lo] <= e0 < row[hi]
        while (hi - lo > 1) {
            const int mid = lo + ((hi - lo) >> 1);
            if ((unsigned)__ldg(row + mid) <= e0)
                lo = mid;
            else
                hi = mid;
        }
        for (int u0 = lo; e0 < e1 && u0 < V; u0 += 32) {
            const int u = u0 + lane;
            const unsigned rs = u < V ? (unsigned)__ldg(row + u) : 0x7fffffffu;
            const unsigned stop = min(e1, (unsigned)__ldg(row + min(u0 + 32, V)));
            for (; e0 < stop; e0 += 32) {
                const unsigned e = e0 + (unsigned)lane;
                const int k = owner_lane(rs, e);  // rows without edges share starts: the last one owns e
                if (e < stop) {
                    const int2 ew = __ldg(adj + e);
                    raw[atomicAdd(cursor + ew.x, 1)] = make_int2(u0 + k, ew.y);
                }
            }
            e0 = stop;
        }
    }
}

// Rows of up to 32 edges: one per warp, ordered by (weight, source).  Weights are not
// negative here, so the packed pair orders as an unsigned 64-bit number.
__global__ void in_sort_short(const int* __restrict__ row, const int* __restrict__ indeg, int V,
                              const int2* __restrict__ raw, int2* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int v = warp; v < V; v += nwarps) {
        const int n = __ldg(indeg + v);
        if (n == 0 || n > 32) continue;
        const int rs = __ldg(row + v);
        unsigned long long key = (unsigned long long)INT_MAX << 32;  // the padding
        if (lane < n) {
            const int2 uw = __ldg(raw + rs + lane);
            key = ((unsigned long long)(unsigned)uw.y << 32) | (unsigned)uw.x;
        }
        for (int k = 2; k < 2 * n && k <= 32; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                const unsigned long long other = __shfl_xor_sync(kFull, key, j);
                const bool lower = (lane & j) == 0, up = (lane & k) == 0;
                key = (lower == up) == (key < other) ? key : other;
            }
        }
        if (lane < padded4(n)) out[rs + lane] = make_int2((int)(unsigned)key, (int)(key >> 32));
    }
}

// Longer rows: one per block, counting sort by weight bucket.
__global__ void __launch_bounds__(kInSortThreads) in_sort_long(const int* __restrict__ row,
                                                               const int* __restrict__ indeg,
                                                               const int* __restrict__ longs, unsigned n_long, int shift,
                                                               const int2* __restrict__ raw, int2* __restrict__ out) {
    __shared__ int hist[kInBuckets];
    constexpr int kPer = kInBuckets / kInSortThreads;
    for (unsigned r = blockIdx.x; r < n_long; r += gridDim.x) {
        const int v = __ldg(longs + r), n = __ldg(indeg + v), rs = __ldg(row + v);
#pragma unroll
        for (int k = 0; k < kPer; ++k) hist[threadIdx.x * kPer + k] = 0;
        __syncthreads();
        for (int i = (int)threadIdx.x; i < n; i += kInSortThreads) atomicAdd(&hist[__ldg(raw + rs + i).y >> shift], 1);
        __syncthreads();
        int h[kPer], sum = 0, total;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            h[k] = hist[threadIdx.x * kPer + k];
            sum += h[k];
        }
        int at = rs + block_exclusive(sum, &total);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            hist[threadIdx.x * kPer + k] = at;
            at += h[k];
        }
        __syncthreads();
        for (int i = (int)threadIdx.x; i < n; i += kInSortThreads) {
            const int2 uw = __ldg(raw + rs + i);
            out[atomicAdd(&hist[uw.y >> shift], 1)] = uw;
        }
        if ((int)threadIdx.x < padded4(n) - n) out[rs + n + (int)threadIdx.x] = make_int2(0, INT_MAX);
        __syncthreads();
    }
}

}  // namespace

void in_rows_free(c2g_graph* g) {
    for (void* p : {(void*)g->in_row, (void*)g->in_adj, (void*)g->in_seg})
        if (p) cudaFree(p);
    g->in_row = nullptr;
    g->in_seg = nullptr;
    g->in_segs = 0;
    g->in_adj = nullptr;
}

// The rows exist when this returns C2G_OK and g->in_adj is set.  A graph they do not serve
// (no edges or no int32 weights, a weight below 0 or above kInMaxWeight, more than 2^31 - 1
// padded edges) or that they do not fit beside simply has none: its queries push.
int build_in_rows(c2g_graph* g) {
    if (!g->adj_w || g->E == 0 || g->in_adj) return C2G_OK;
    const size_t V = (size_t)g->V, E = (size_t)g->E;
    const int scan_blocks = (int)((V + kScanThreads * kScanItems - 1) / (kScanThreads * kScanItems));
    // one temporary: stats | in-degrees | cursors | long rows | scan block sums
    const size_t words = V * 3 + (size_t)scan_blocks;
    char* tmp = nullptr;
    int2* raw = nullptr;
    cudaError_t e = cudaMalloc(&tmp, 256 + sizeof(int) * words);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return C2G_OK;
    }
    InStats* st = reinterpret_cast<InStats*>(tmp);
    int* indeg = reinterpret_cast<int*>(tmp + 256);
    int *cursor = indeg + V, *longs = cursor + V, *sums = longs + V;
    InStats h{INT_MAX, INT_MIN, 0u, 0u, 0ull};
    const int blocks = g->num_sms * 8;
    e = cudaMemsetAsync(indeg, 0, sizeof(int) * V, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(st, &h, sizeof(h), cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) {
        in_count<<<blocks, 256, 0, g->stream>>>(g->adj_w, (unsigned)E, indeg, st);
        in_scan_blocks<<<scan_blocks, kScanThreads, 0, g->stream>>>(indeg, g->V, sums, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    const bool usable = e == cudaSuccess && h.wmin >= 0 && h.wmax <= kInMaxWeight && h.padded < (1ull << 31);
    bool fits = usable;
    if (usable) {
        fits = cudaMalloc(&g->in_row, sizeof(int) * (V + 1)) == cudaSuccess &&
               cudaMalloc(&g->in_adj, sizeof(int2) * (size_t)h.padded) == cudaSuccess &&
               cudaMalloc(&raw, sizeof(int2) * (size_t)h.padded) == cudaSuccess;
        if (!fits) cudaGetLastError();
    }
    if (fits) {
        int shift = 0;
        while ((h.wmax >> shift) >= kInBuckets) ++shift;
        in_scan_sums<<<1, kScanThreads, 0, g->stream>>>(sums, scan_blocks);
        in_scan_rows<<<scan_blocks, kScanThreads, 0, g->stream>>>(indeg, g->V, sums, g->in_row, cursor, longs, st);
        in_scatter<<<blocks, 256, 0, g->stream>>>(g->row, g->adj_w, g->V, (unsigned)E, cursor, raw);
        in_sort_short<<<blocks, 256, 0, g->stream>>>(g->in_row, indeg, g->V, raw, g->in_adj);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
        if (e == cudaSuccess && h.n_long) {
            in_sort_long<<<blocks, kInSortThreads, 0, g->stream>>>(g->in_row, indeg, longs, h.n_long, shift, raw,
                                                                  g->in_adj);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess && h.n_seg) {
            fits = cudaMalloc(&g->in_seg, sizeof(int2) * (size_t)h.n_seg) == cudaSuccess;
            if (!fits) cudaGetLastError();
            if (fits) e = cudaMemsetAsync(&st->n_long, 0, sizeof(unsigned), g->stream);
            if (fits && e == cudaSuccess) {
                in_segments<<<blocks, 256, 0, g->stream>>>(g->in_row, longs, h.n_long, &st->n_long, h.n_seg, g->in_seg);
                e = cudaGetLastError();
            }
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
        g->in_segs = h.n_seg;
        g->in_shift = shift;
        g->in_edges = (int64_t)h.padded;
    }
    if (raw) cudaFree(raw);
    cudaFree(tmp);
    if (e != cudaSuccess || !fits) in_rows_free(g);
    C2G_CUDA(e);
    return C2G_OK;
}

}  // namespace c2g
