// PPR adjoint for sm_103a: gradient of L = sum_{t in T} pi_s(t) with respect to every
// flist edge weight.
//
// With the reference's convention (pr += alpha*r, push (1-alpha)*r*w,
// src/ppr/base/Main.cu:146-150 and :288), pi = alpha * (I - (1-alpha) P^T)^{-1} e_s for
// P[u][v] = w(u,v).  Then
//     dL/dw(u,v) = (1-alpha) * pi(u) * lambda(v),  lambda = (I - (1-alpha) P)^{-1} 1_T.
// lambda is the fixed point of lambda(u) = 1_T(u) + (1-alpha) sum_v w(u,v) lambda(v),
// computed by a transposed push: the same BSP push kernel, run on the reverse CSR
// (in-edges carrying w(u,v)) from the target set, absorbing 1*r instead of alpha*r.
// The gradient pass reads each forward edge once: 12 bytes per edge + 8 per vertex.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

namespace c2g {

// grad[e] = c * pi[u] * lambda[col[e]] for every forward edge e = (u -> col[e]).  Warps
// take tiles of 2^kPullTileLog edges; a tile's first owner comes from the forward tile
// markers (one load), the next 32 owners' row bounds and pi values one per lane, and each
// edge's owner from a shuffle search.  Edges are read 32 at a time, kGradUnroll batches in
// flight, so the lambda gathers of a warp overlap.
constexpr int kGradUnroll = 4;

__global__ void adjoint_grad_kernel(const int* __restrict__ row, const int2* __restrict__ adj,
                                    const int* __restrict__ mark, int V, unsigned E, const float* __restrict__ pi,
                                    const float* __restrict__ lam, float c, float* __restrict__ grad,
                                    int* __restrict__ flags) {
    const int lane = threadIdx.x & 31;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned tw = 1u << kPullTileLog;
    const unsigned ntiles = (E + tw - 1) >> kPullTileLog;
    for (unsigned t = warp; t < ntiles; t += nwarps) {
        unsigned e0 = t << kPullTileLog;
        const unsigned e1 = min(e0 + tw, E);
        unsigned o = (unsigned)__ldg(mark + t);
        while (e0 < e1) {
            const unsigned j = o + (unsigned)lane;
            unsigned base = 0x7fffffffu, endv = 0xffffffffu;
            float pj = 0.f;
            if (j < (unsigned)V) {
                base = (unsigned)__ldg(row + j);
                endv = (unsigned)__ldg(row + j + 1);
                pj = __ldg(pi + j);
            }
            if (o >= (unsigned)V || (unsigned)__shfl_sync(kFull, (int)base, 0) > e0) {
                if (lane == 0) atomicOr(flags, C2G_FLAG_BOUNDS);
                break;
            }
            const unsigned seg_end = min(e1, (unsigned)__shfl_sync(kFull, endv, 31));
            if (seg_end <= e0) {  // 32 owners without edges here (o grows to V at most)
                o += 32;
                continue;
            }
            for (unsigned eb = e0; eb < seg_end; eb += 32u * kGradUnroll) {
                int2 ew[kGradUnroll];
                float pk[kGradUnroll];
#pragma unroll
                for (int u = 0; u < kGradUnroll; ++u) {
                    const unsigned e = eb + (unsigned)lane + 32u * u;
                    pk[u] = __shfl_sync(kFull, pj, owner_lane(base, e));
                    ew[u] = e < seg_end ? __ldg(adj + e) : make_int2(0, 0);
                }
#pragma unroll
                for (int u = 0; u < kGradUnroll; ++u) {
                    const unsigned e = eb + (unsigned)lane + 32u * u;
                    if (e < seg_end) grad[e] = c * pk[u] * __ldg(lam + ew[u].x);
                }
            }
            e0 = seg_end;
            o += 32;
        }
    }
}

// out[i] = pi[v[i]]: what the loss needs of pi.
__global__ void adjoint_at_targets(const float* __restrict__ pi, const int* __restrict__ v, int n, float* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = __ldg(pi + __ldg(v + i));
}

// Per-handle workspace of the gradient, kept across calls: a training loop calls it every step, and
// allocating and freeing its arrays each time (cudaFree waits for the device) took 0.9 ms of a call at
// scale 20.
struct AdjointWork {
    float *pi = nullptr, *lam = nullptr;  // [V]
    float* grad = nullptr;                // [E], once a gradient goes to the host
    int32_t* tv = nullptr;                // distinct targets,
    float *tr = nullptr, *tpi = nullptr;  // their multiplicities, and pi there
    size_t targets = 0;                   // allocated
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaStream_t beside = nullptr;        // copies while the pushes run
};

void adjoint_free(c2g_graph* g) {
    AdjointWork* w = reinterpret_cast<AdjointWork*>(g->adjoint);
    if (!w) return;
    for (void* p : {(void*)w->pi, (void*)w->lam, (void*)w->grad, (void*)w->tv, (void*)w->tr, (void*)w->tpi})
        if (p) cudaFree(p);
    for (cudaEvent_t ev : {w->ev0, w->ev1})
        if (ev) cudaEventDestroy(ev);
    if (w->beside) cudaStreamDestroy(w->beside);
    delete w;
    g->adjoint = nullptr;
}

static int adjoint_alloc(c2g_graph* g, size_t targets, bool host_grad, AdjointWork** out) {
    AdjointWork* w = reinterpret_cast<AdjointWork*>(g->adjoint);
    if (!w) g->adjoint = w = new AdjointWork();
    const size_t V = (size_t)g->V, E = (size_t)g->E;
    cudaError_t e = cudaSuccess;
    if (!w->ev0) e = cudaEventCreate(&w->ev0);
    if (e == cudaSuccess && !w->ev1) e = cudaEventCreate(&w->ev1);
    if (e == cudaSuccess && host_grad && !w->beside) e = cudaStreamCreateWithFlags(&w->beside, cudaStreamNonBlocking);
    if (e == cudaSuccess && !w->pi) e = cudaMalloc(&w->pi, sizeof(float) * V);
    if (e == cudaSuccess && !w->lam) e = cudaMalloc(&w->lam, sizeof(float) * V);
    if (e == cudaSuccess && host_grad && !w->grad) e = cudaMalloc(&w->grad, sizeof(float) * (E ? E : 1));
    if (e == cudaSuccess && w->targets < targets) {
        for (void* p : {(void*)w->tv, (void*)w->tr, (void*)w->tpi})
            if (p) cudaFree(p);
        w->tv = nullptr;
        w->tr = w->tpi = nullptr;
        w->targets = 0;
        e = cudaMalloc(&w->tv, sizeof(int32_t) * targets);
        if (e == cudaSuccess) e = cudaMalloc(&w->tr, sizeof(float) * targets);
        if (e == cudaSuccess) e = cudaMalloc(&w->tpi, sizeof(float) * targets);
        if (e == cudaSuccess) w->targets = targets;
    }
    if (e != cudaSuccess) adjoint_free(g);
    C2G_CUDA(e);
    *out = w;
    return C2G_OK;
}

int set_float_weights(c2g_graph* g, const float* w, int on_device);

// Maps the pages inside a host array that a copy will fill, without writing to it (where the system cannot, the copy
// maps them).
static void map_pages(void* p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = ((uintptr_t)p + page - 1) & ~(page - 1),
                    b = ((uintptr_t)p + bytes) & ~(page - 1);
    if (p && a < b) madvise(reinterpret_cast<void*>(a), b - a, MADV_POPULATE_WRITE);
#else
    (void)p, (void)bytes;
#endif
}

// Lets the driver make the pages of a large host array ready for a copy, by reading them into `scratch` (0.8 ms of
// the first copy on 40 to 60 MB of mapped pages that no copy has touched).  Returns when it is done; what fails here
// is left to the copy itself.
constexpr size_t kReadyBytes = 4u << 20;
static void ready_pages(const void* p, size_t bytes, void* scratch, size_t room, cudaStream_t s) {
    if (!p || bytes < kReadyBytes || room < kReadyBytes) return;
    bool ok = true;
    for (size_t at = 0; at < bytes && ok; at += room)
        ok = cudaMemcpyAsync(scratch, (const char*)p + at, std::min(room, bytes - at), cudaMemcpyHostToDevice, s) ==
             cudaSuccess;
    if (cudaStreamSynchronize(s) != cudaSuccess || !ok) cudaGetLastError();
}

}  // namespace c2g

using namespace c2g;

extern "C" int c2g_ppr_adjoint(c2g_graph* g, int32_t source, const c2g_ppr_params* params, int32_t n_targets,
                               const int32_t* targets, float rmax_backward, float* grad, float* pi_out,
                               float* lambda_out, double* loss, int on_device, c2g_stats* stats) {
    if (!g || !params || !targets || !grad) return fail(C2G_ERR_ARG, "NULL argument");
    if (source < 0 || source >= g->V) return fail(C2G_ERR_RANGE, "source %d out of range [0,%d)", source, g->V);
    if (n_targets < 1) return fail(C2G_ERR_ARG, "need at least one target");
    if (!(params->alpha > 0.f && params->alpha < 1.f)) return fail(C2G_ERR_ARG, "alpha must be in (0,1)");
    if (params->seeded) return fail(C2G_ERR_UNSUPPORTED, "the adjoint differentiates the base push");
    if (!(rmax_backward >= 0.f)) return fail(C2G_ERR_ARG, "rmax_backward must be >= 0");
    if (!g->adj_f) return fail(C2G_ERR_UNSUPPORTED, "graph has no float weights (flist)");
    // distinct targets, each with its multiplicity as the initial residual
    std::vector<int32_t> tv;
    std::vector<float> tr;
    {
        std::vector<int32_t> sorted(targets, targets + n_targets);
        for (int32_t t : sorted)
            if (t < 0 || t >= g->V) return fail(C2G_ERR_RANGE, "target %d out of range", t);
        std::sort(sorted.begin(), sorted.end());
        for (size_t i = 0; i < sorted.size(); ++i) {
            if (tv.empty() || tv.back() != sorted[i]) {
                tv.push_back(sorted[i]);
                tr.push_back(1.0f);
            } else {
                tr.back() += 1.0f;
            }
        }
    }
    std::lock_guard<std::mutex> lk(g->mu);
    struct Scope {
        int prev = -1;
        explicit Scope(int d) {
            cudaGetDevice(&prev);
            cudaSetDevice(d);
        }
        ~Scope() {
            if (prev >= 0) cudaSetDevice(prev);
        }
    } scope(g->device);
    const size_t V = (size_t)g->V, E = (size_t)g->E;
    AdjointWork* w = nullptr;
    int rc = with_room_of_rows(g, [&] {
        int r = build_reverse_graph(g);
        if (!r) r = build_row_lists(g, g->row, g->row_r, &g->rows_out);
        return r ? r : adjoint_alloc(g, tv.size(), !on_device, &w);
    });
    if (rc) return rc;
    float *const pi = w->pi, *const lam = w->lam, *const dgrad = on_device ? grad : w->grad;
    float ms_f = 0.f, ms_b = 0.f, ms_g = 0.f;
    TraversalCtl cf, cb;
    cudaError_t e = cudaMemcpyAsync(w->tv, tv.data(), sizeof(int32_t) * tv.size(), cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(w->tr, tr.data(), sizeof(float) * tr.size(), cudaMemcpyHostToDevice, g->stream);
    C2G_CUDA(e);
    // forward: pi
    c2g_ppr_params fp = *params;
    fp.r0 = 1.0f;
    fp.pr0 = fp.alpha;
    rc = with_room_of_rows(g, [&] {
        return ppr_launch_view(g, g->row, g->adj_f, g->row_r, g->adj_r, g->rows_in, source, fp, fp.alpha, 0, nullptr,
                               nullptr, nullptr, nullptr, 0, pi, nullptr, nullptr);
    });
    // Nothing is written to the caller's arrays before both pushes have ended well.  Their pages are mapped beside
    // the forward push and made ready beside the backward one: a copy after them that has to do both takes 2 ms
    // longer on 40 MB.
    if (!rc && !on_device) {
        map_pages(grad, sizeof(float) * E);
        map_pages(pi_out, sizeof(float) * V);
        map_pages(lambda_out, sizeof(float) * V);
    }
    if (!rc && (cudaMemcpyAsync(&cf, g->ppr.ctl, sizeof(cf), cudaMemcpyDeviceToHost, g->stream) != cudaSuccess ||
                cudaStreamSynchronize(g->stream) != cudaSuccess ||
                cudaEventElapsedTime(&ms_f, g->ev0, g->ev1) != cudaSuccess))
        rc = fail(C2G_ERR_CUDA, "adjoint: reading the forward push status failed");
    // backward: lambda, transposed push from the targets, absorbing the whole residual
    c2g_ppr_params bp = *params;
    bp.rmax = rmax_backward;
    if (!rc)
        rc = ppr_launch_view(g, g->row_r, g->adj_r, g->row, g->adj_f, g->rows_out, tv[0], bp, 1.0f, (int32_t)tv.size(),
                             w->tv, w->tr, nullptr, nullptr, 0, lam, nullptr, nullptr);
    if (rc) return rc;
    if (!on_device) {
        ready_pages(grad, sizeof(float) * E, w->grad, sizeof(float) * E, w->beside);
        ready_pages(pi_out, sizeof(float) * V, w->grad, sizeof(float) * E, w->beside);
        ready_pages(lambda_out, sizeof(float) * V, w->grad, sizeof(float) * E, w->beside);
    }
    e = cudaMemcpyAsync(&cb, g->ppr.ctl, sizeof(cb), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms_b, g->ev0, g->ev1);
    C2G_CUDA(e);
    if ((cf.flags | cb.flags) & (C2G_FLAG_BARRIER_TIMEOUT | C2G_FLAG_QUEUE_OVERFLOW | C2G_FLAG_BOUNDS))
        return fail(C2G_ERR_OVERFLOW, "adjoint push reported device errors (flags %d/%d)", cf.flags, cb.flags);
    // gradient pass
    cudaEventRecord(w->ev0, g->stream);
    if (E)
        adjoint_grad_kernel<<<g->num_sms * 8, 256, 0, g->stream>>>(g->row, g->adj_f, g->mark_f, g->V, (unsigned)E, pi,
                                                                   lam, 1.0f - params->alpha, dgrad,
                                                                   &g->ppr.ctl->flags);
    cudaEventRecord(w->ev1, g->stream);
    e = cudaGetLastError();
    if (e == cudaSuccess && !on_device)
        e = cudaMemcpyAsync(grad, dgrad, sizeof(float) * E, cudaMemcpyDeviceToHost, g->stream);
    std::vector<float> tpi(loss ? tv.size() : 0);
    if (e == cudaSuccess && loss) {
        adjoint_at_targets<<<(int)std::min<size_t>((tv.size() + 255) / 256, 1024), 256, 0, g->stream>>>(
            pi, w->tv, (int)tv.size(), w->tpi);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(tpi.data(), w->tpi, sizeof(float) * tv.size(), cudaMemcpyDeviceToHost, g->stream);
    }
    if (e == cudaSuccess && pi_out)
        e = cudaMemcpyAsync(pi_out, pi, sizeof(float) * V, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                            g->stream);
    if (e == cudaSuccess && lambda_out)
        e = cudaMemcpyAsync(lambda_out, lam, sizeof(float) * V,
                            on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, g->stream);
    int gflags = 0;  // the gradient pass's bounds checks report into the push's control block
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&gflags, &g->ppr.ctl->flags, sizeof(int), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    C2G_CUDA(e);
    C2G_CUDA(cudaEventElapsedTime(&ms_g, w->ev0, w->ev1));
    if (gflags & C2G_FLAG_BOUNDS) return fail(C2G_ERR_OVERFLOW, "adjoint gradient pass: device index check failed");
    if (loss) {
        double L = 0.0;
        for (int32_t t = 0; t < n_targets; ++t)
            L += (double)tpi[(size_t)(std::lower_bound(tv.begin(), tv.end(), targets[t]) - tv.begin())];
        *loss = L;
    }
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->source = source;
        stats->iterations = cf.iterations + cb.iterations;
        stats->vertices_popped = cf.popped + cb.popped;
        stats->edges_relaxed = cf.relaxed + cb.relaxed;
        stats->touched = cf.touched + cb.touched;
        stats->n_seeds = (int64_t)tv.size();
        stats->device_ms = ms_f + ms_b + ms_g;
        stats->status_flags = cf.flags | cb.flags;
        // two pushes (12V + 20F + 12R each) + the gradient pass (12E + 8V)
        stats->alg_bytes = 24.0 * V + 20.0 * (double)(cf.popped + cb.popped) + 12.0 * (double)(cf.relaxed + cb.relaxed) +
                           12.0 * (double)E + 8.0 * (double)V;
    }
    return C2G_OK;
}

extern "C" int c2g_graph_set_weights(c2g_graph* g, const float* flist, int on_device) {
    if (!g || !flist) return fail(C2G_ERR_ARG, "NULL argument");
    std::lock_guard<std::mutex> lk(g->mu);
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    const int rc = set_float_weights(g, flist, on_device);
    if (prev >= 0) cudaSetDevice(prev);
    return rc;
}
