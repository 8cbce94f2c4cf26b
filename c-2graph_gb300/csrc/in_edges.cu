// In-edges of a graph, built on the device: rows ordered by int32 weight for the SSSP pull
// rounds (sssp.cu, batch.cu), and the reverse CSR with float weights and its rows by length for
// the push kernels' pull rounds (ppr.cu, batch.cu, adsorption.cu, adjoint.cu).
//
// Rows ordered by weight: row v holds v's in-edges (source, weight) in ascending order of weight, padded with
// (0, INT_MAX) to a multiple of 4 edges, so that a row is read in aligned 32-byte groups and
// a reader can stop at the first group whose weights cannot improve v any more.  The
// reference has no in-edges; it relaxes out-edges only (src/sssp/purn/Main.cu:236-331).
//
// They are built when the graph is made, or by its first SSSP call where it has both kinds of weights (int32 weights
// never change): count the in-edges, scan the padded row lengths, scatter the edges into their rows, order each row.
// Rows of up to 32 edges are ordered by a warp (bitonic network on weight and source), longer
// ones by a block (counting sort over kInBuckets buckets of weight).  A bucket spans 2^shift
// weights, where 2^shift * kInBuckets covers the largest weight; inside a bucket the order is
// free, so a reader compares with the bucket's lower end, (w >> shift) << shift.  Each step is
// bound by scattered 8-byte accesses: at scale 22 (65M edges) making the graph from host
// arrays takes 68.2 ms with the rows and 63.5 ms without.
#include <algorithm>
#include <climits>
#include <cstdint>

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
    unsigned n_hub;              // rows of more than 256 edges
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
__device__ __forceinline__ int padded(int n, int pad) { return pad ? padded4(n) : n; }

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

// Edges (padded to 4 when pad) of each scan block's rows (the padded sum may pass 2^31: st->padded).
__global__ void __launch_bounds__(kScanThreads) in_scan_blocks(const int* __restrict__ indeg, int V, int pad,
                                                              int* __restrict__ block_sum, InStats* st) {
    const int base = (int)blockIdx.x * kScanThreads * kScanItems;
    int n = 0;
    for (int k = 0; k < kScanItems; ++k) {
        const int v = base + k * kScanThreads + (int)threadIdx.x;
        if (v < V) n += padded(__ldg(indeg + v), pad);
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

// Row starts, the scatter's cursors and, when padded, the list of rows longer than a warp.
__global__ void __launch_bounds__(kScanThreads) in_scan_rows(const int* __restrict__ indeg, int V, int pad,
                                                            const int* __restrict__ block_sum, int* __restrict__ row,
                                                            int* __restrict__ cursor, int* __restrict__ longs,
                                                            InStats* st) {
    const int base = ((int)blockIdx.x * kScanThreads + (int)threadIdx.x) * kScanItems;
    int d[kScanItems], n = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        d[k] = base + k < V ? __ldg(indeg + base + k) : 0;
        n += padded(d[k], pad);
    }
    int total;
    int at = block_sum[blockIdx.x] + block_exclusive(n, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int v = base + k;
        const bool lng = pad && v < V && d[k] > 32;
        if (lng && d[k] > 256) atomicAdd(&st->n_hub, 1u);
        if (lng && padded4(d[k]) > kInHead)
            atomicAdd(&st->n_seg, (unsigned)(padded4(d[k]) - kInHead + kInSegment - 1) / kInSegment);
        if (v < V) {
            row[v] = at;
            cursor[v] = at;
        }
        at += padded(d[k], pad);
        if (v == V - 1) row[V] = at;
        if (pad) list_push(longs, &st->n_long, (unsigned)V, reinterpret_cast<int*>(&st->n_long), lng, v);
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

// Row starts of a CSR by chunk of 32 edges: bit e % 32 of bits[e / 32] says that edge e starts a row.
__global__ void start_bits(const int* __restrict__ row, int V, unsigned* __restrict__ bits) {
    const int stride = gridDim.x * blockDim.x;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += stride) {
        const int rs = __ldg(row + v);
        if (__ldg(row + v + 1) > rs) atomicOr(bits + (rs >> 5), 1u << (rs & 31));
    }
}

__global__ void start_counts(const unsigned* __restrict__ bits, int n, int* __restrict__ count) {
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) count[i] = __popc(__ldg(bits + i));
}

// The non-empty rows in order, from the starts before each chunk.
__global__ void start_rows(const int* __restrict__ row, int V, const unsigned* __restrict__ bits,
                           const int* __restrict__ prefix, int* __restrict__ rows) {
    const int stride = gridDim.x * blockDim.x;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += stride) {
        const int rs = __ldg(row + v);
        if (__ldg(row + v + 1) > rs)
            rows[__ldg(prefix + (rs >> 5)) + __popc(__ldg(bits + (rs >> 5)) & ((1u << (rs & 31)) - 1u))] = v;
    }
}

// Class of a row of n edges (RowLists).
__device__ __forceinline__ int row_class(int n) {
    int c = 0;
#pragma unroll
    for (int k = 1; k < kRowClasses; ++k)
        if (n <= ((32 * kLaneEdges) >> (k - 1))) c = k;
    return c;
}

struct ClassCount {
    unsigned n[kRowClasses];  // records
    unsigned n_long;          // rows of class 0
};

// Records per class (fill = false), or the records themselves, appended from `at` on.
template <bool kFill>
__global__ void __launch_bounds__(256) row_classes(const int* __restrict__ row, const int* __restrict__ other, int V,
                                                  int segment, ClassCount* count, int4* __restrict__ rec, int2* __restrict__ seg) {
    __shared__ unsigned s_n[kRowClasses], s_at[kRowClasses];
    for (int v0 = (int)(blockIdx.x * blockDim.x); v0 < V; v0 += (int)(gridDim.x * blockDim.x)) {
        if (threadIdx.x < kRowClasses) s_n[threadIdx.x] = 0u;
        __syncthreads();
        const int v = v0 + (int)threadIdx.x;
        const int rs = v < V ? __ldg(row + v) : 0, n = v < V ? __ldg(row + v + 1) - rs : 0;
        const int c = row_class(n);
        const unsigned parts = n == 0 ? 0u : c == 0 ? (unsigned)(n + segment - 1) / (unsigned)segment : 1u;
        unsigned at = 0u;
        if (parts) at = atomicAdd(&s_n[c], parts);
        __syncthreads();
        if (threadIdx.x < kRowClasses && s_n[threadIdx.x])
            s_at[threadIdx.x] = atomicAdd(&count->n[threadIdx.x], s_n[threadIdx.x]);
        __syncthreads();
        if (kFill && parts) {
            const int out = __ldg(other + v + 1) - __ldg(other + v);
            at += s_at[c];
            if (c) {
                rec[at] = make_int4(v, rs, n, out);
            } else {
                const int id = (int)atomicAdd(&count->n_long, 1u);
                for (unsigned k = 0; k < parts; ++k) {
                    rec[at + k] = make_int4(v, rs + (int)k * segment, min(segment, n - (int)k * segment), out);
                    seg[at + k] = make_int2(id, (int)parts);
                }
            }
        } else if (!kFill && parts && c == 0) {
            atomicAdd(&count->n_long, 1u);
        }
        __syncthreads();
    }
}

}  // namespace

void row_lists_free(RowLists& r) {
    for (void* p : {(void*)r.rec, (void*)r.seg})
        if (p) cudaFree(p);
    r = RowLists();
}

// The non-empty rows of a CSR by length; `other` is the CSR of the opposite direction.
int build_row_lists(c2g_graph* g, const int* row, const int* other, RowLists* out) {
    if (out->rec || g->E == 0) return C2G_OK;
    ClassCount h{};
    ClassCount* d = nullptr;
    C2G_CUDA(cudaMalloc(&d, sizeof(ClassCount)));
    const int blocks = std::min(g->num_sms * 8, (g->V + 255) / 256);
    RowLists r;
    // a segment is one step of a warp (256 edges) where every round is latency, two where it is throughput
    r.segment = g->E <= kShortSegmentEdges ? 32 * kLaneEdges : 64 * kLaneEdges;
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(ClassCount), g->stream);
    if (e == cudaSuccess) {
        row_classes<false><<<blocks, 256, 0, g->stream>>>(row, other, g->V, r.segment, d, nullptr, nullptr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    unsigned total = 0, unit = 0;
    for (int c = 0; c < kRowClasses; ++c) {
        const unsigned rows = c <= 1 ? 1u : 1u << (c - 1);  // rows a warp takes at a time
        r.n[c] = h.n[c];
        r.off[c] = total;
        r.unit[c] = unit;
        total += h.n[c];
        unit += (h.n[c] + rows - 1) / rows;
    }
    r.unit[kRowClasses] = unit;
    r.n_long = h.n_long;
    if (e == cudaSuccess) e = cudaMalloc(&r.rec, sizeof(int4) * (total ? total : 1));
    if (e == cudaSuccess) e = cudaMalloc(&r.seg, sizeof(int2) * (h.n[0] ? h.n[0] : 1));
    if (e == cudaSuccess) {
        ClassCount at{};
        for (int c = 0; c < kRowClasses; ++c) at.n[c] = r.off[c];
        e = cudaMemcpyAsync(d, &at, sizeof(at), cudaMemcpyHostToDevice, g->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);  // `at` is read
    }
    if (e == cudaSuccess) {
        row_classes<true><<<blocks, 256, 0, g->stream>>>(row, other, g->V, r.segment, d, r.rec, r.seg);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    cudaFree(d);
    if (e != cudaSuccess) row_lists_free(r);
    C2G_CUDA(e);
    *out = r;
    return C2G_OK;
}

// Scatter the float-weighted out-edges into the reverse CSR's rows (in any order within a row); cursor: V ints.
static cudaError_t scatter_reverse(c2g_graph* g, const int2* fwd, int* cursor) {
    const size_t V = (size_t)g->V;
    cudaError_t e = cudaMemcpyAsync(cursor, g->row_r, sizeof(int) * V, cudaMemcpyDeviceToDevice, g->stream);
    if (e == cudaSuccess && g->E) {
        in_scatter<<<g->num_sms * 8, 256, 0, g->stream>>>(g->row, fwd, g->V, (unsigned)g->E, cursor, g->adj_r);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    return e;
}

static int build_row_starts(c2g_graph* g);

// Reverse CSR of the float-weighted graph (in-edges carrying w(u,v)), its rows by length and by
// chunk, the forward CSR's tile owners; built when the graph is made, where it has float weights only, else on first use.
int build_reverse_graph(c2g_graph* g) {
    if (g->adj_r) return C2G_OK;
    const int2* fwd = g->adj_f ? g->adj_f : g->adj_w;  // float weights when the graph has them
    if (!fwd) return fail(C2G_ERR_UNSUPPORTED, "graph has no edge weights");
    const size_t V = (size_t)g->V, E = (size_t)g->E;
    const int scan_blocks = (int)((V + kScanThreads * kScanItems - 1) / (kScanThreads * kScanItems));
    char* tmp = nullptr;  // stats | in-degrees | cursors | scan block sums
    C2G_CUDA(cudaMalloc(&tmp, 256 + sizeof(int) * (V * 2 + (size_t)scan_blocks + 1)));
    InStats* st = reinterpret_cast<InStats*>(tmp);
    int* indeg = reinterpret_cast<int*>(tmp + 256);
    int *cursor = indeg + V, *sums = cursor + V;
    cudaError_t e = cudaMalloc(&g->row_r, sizeof(int) * (V + 1));
    if (e == cudaSuccess) e = cudaMalloc(&g->adj_r, sizeof(int2) * (E ? E : 1));
    if (e == cudaSuccess) e = cudaMemsetAsync(tmp, 0, 256 + sizeof(int) * V, g->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(g->row_r, 0, sizeof(int) * (V + 1), g->stream);
    if (e == cudaSuccess && E) {
        in_count<<<g->num_sms * 8, 256, 0, g->stream>>>(fwd, (unsigned)E, indeg, st);
        in_scan_blocks<<<scan_blocks, kScanThreads, 0, g->stream>>>(indeg, g->V, 0, sums, st);
        in_scan_sums<<<1, kScanThreads, 0, g->stream>>>(sums, scan_blocks);
        in_scan_rows<<<scan_blocks, kScanThreads, 0, g->stream>>>(indeg, g->V, 0, sums, g->row_r, cursor, nullptr, st);
        e = cudaGetLastError();
    }
    InStats h{};
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = scatter_reverse(g, fwd, cursor);
    cudaFree(tmp);
    if (e == cudaSuccess && g->adj_f) {  // the largest positive weight: positive floats order as integers
        g->wstat_wmax_bits = (uint32_t)h.wmax;
        g->wstat_valid = true;
    }
    int rc = C2G_OK;
    if (e != cudaSuccess)
        rc = fail(e == cudaErrorMemoryAllocation ? C2G_ERR_OOM : C2G_ERR_CUDA, "reverse CSR: %s", cudaGetErrorString(e));
    if (!rc) rc = build_markers(g, g->row, &g->mark_f);
    if (!rc) rc = build_row_lists(g, g->row_r, g->row, &g->rows_in);
    if (!rc) rc = build_row_starts(g);
    if (rc) {
        cudaGetLastError();
        reverse_free(g);
    }
    return rc;
}

// Row starts of the reverse CSR by chunk.
static int build_row_starts(c2g_graph* g) {
    const size_t V = (size_t)g->V, n = ((size_t)g->E + 31) / 32;
    if (n == 0) return C2G_OK;
    const int scan_blocks = (int)((n + kScanThreads * kScanItems - 1) / (kScanThreads * kScanItems));
    int* tmp = nullptr;  // counts | cursors (unused) | scan block sums | stats
    C2G_CUDA(cudaMalloc(&tmp, sizeof(int) * (2 * n + (size_t)scan_blocks) + 256));
    int *count = tmp, *cursor = tmp + n, *sums = cursor + n;
    cudaError_t e = cudaMalloc(&g->r_bits, sizeof(unsigned) * n);
    if (e == cudaSuccess) e = cudaMalloc(&g->r_prefix, sizeof(int) * (n + 1));
    if (e == cudaSuccess) e = cudaMalloc(&g->r_rows, sizeof(int) * V);
    if (e == cudaSuccess) e = cudaMemsetAsync(g->r_bits, 0, sizeof(unsigned) * n, g->stream);
    if (e == cudaSuccess) {
        InStats* st = reinterpret_cast<InStats*>((reinterpret_cast<uintptr_t>(sums + scan_blocks) + 63) & ~(uintptr_t)63);
        const int blocks = g->num_sms * 8;
        start_bits<<<blocks, 256, 0, g->stream>>>(g->row_r, g->V, g->r_bits);
        start_counts<<<blocks, 256, 0, g->stream>>>(g->r_bits, (int)n, count);
        in_scan_blocks<<<scan_blocks, kScanThreads, 0, g->stream>>>(count, (int)n, 0, sums, st);
        in_scan_sums<<<1, kScanThreads, 0, g->stream>>>(sums, scan_blocks);
        in_scan_rows<<<scan_blocks, kScanThreads, 0, g->stream>>>(count, (int)n, 0, sums, g->r_prefix, cursor, nullptr, st);
        start_rows<<<blocks, 256, 0, g->stream>>>(g->row_r, g->V, g->r_bits, g->r_prefix, g->r_rows);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    cudaFree(tmp);
    C2G_CUDA(e);
    return C2G_OK;
}

// New float weights: the reverse CSR's rows stay, their edges are written anew (cursor: V ints, where there is a
// reverse CSR).  If that fails it goes, and with it what holds its addresses; the next call that needs it builds it.
int refresh_reverse_graph(c2g_graph* g, int* cursor) {
    g->wstat_valid = false;
    if (!g->adj_r) return C2G_OK;
    const cudaError_t e = scatter_reverse(g, g->adj_f, cursor);
    if (e != cudaSuccess) {
        ads_free(g);
        reverse_free(g);
    }
    C2G_CUDA(e);
    return C2G_OK;
}

void reverse_free(c2g_graph* g) {
    for (void* p : {(void*)g->row_r, (void*)g->adj_r, (void*)g->mark_f, (void*)g->r_bits,
                    (void*)g->r_prefix, (void*)g->r_rows})
        if (p) cudaFree(p);
    g->r_bits = nullptr;
    g->r_prefix = nullptr;
    g->r_rows = nullptr;
    row_lists_free(g->rows_in);
    row_lists_free(g->rows_out);
    g->wstat_valid = false;
    g->row_r = nullptr;
    g->adj_r = nullptr;
    g->mark_f = nullptr;
}

int ensure_reverse(c2g_graph* g) {
    if (g->borrowed || g->reverse_tried || g->adj_r) return C2G_OK;
    g->reverse_tried = true;
    const int rc = build_reverse_graph(g);
    return rc == C2G_ERR_OOM ? C2G_OK : rc;
}

int ensure_in_rows(c2g_graph* g) {
    if (g->borrowed || g->in_rows_tried || g->in_adj) return C2G_OK;
    g->in_rows_tried = true;
    return build_in_rows(g);
}

// Free them where no view shares them; false: there was nothing to free.
bool in_rows_drop(c2g_graph* g) {
    if (g->borrowed || !g->in_adj || *g->views > 0) return false;
    in_rows_free(g);
    return true;
}

bool reverse_drop(c2g_graph* g) {
    if (g->borrowed || !g->adj_r || *g->views > 0) return false;
    ads_free(g);  // its captured launches hold the addresses
    reverse_free(g);
    return true;
}

void in_rows_free(c2g_graph* g) {
    for (void* p : {(void*)g->in_row, (void*)g->in_adj, (void*)g->in_seg})
        if (p) cudaFree(p);
    g->in_row = nullptr;
    g->in_seg = nullptr;
    g->in_segs = 0;
    g->in_hubs = false;
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
    InStats h{INT_MAX, INT_MIN, 0u, 0u, 0u, 0ull};
    const int blocks = g->num_sms * 8;
    e = cudaMemsetAsync(indeg, 0, sizeof(int) * V, g->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(st, &h, sizeof(h), cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) {
        in_count<<<blocks, 256, 0, g->stream>>>(g->adj_w, (unsigned)E, indeg, st);
        in_scan_blocks<<<scan_blocks, kScanThreads, 0, g->stream>>>(indeg, g->V, 1, sums, st);
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
        in_scan_rows<<<scan_blocks, kScanThreads, 0, g->stream>>>(indeg, g->V, 1, sums, g->in_row, cursor, longs, st);
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
        g->in_hubs = h.n_hub > 0u;
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
