// Degree ordering of an oriented edge relation.
//
// When every edge (u, v) of a self-joined relation has 0 <= u < v, the
// triangles (and 4-cliques) of the join in attribute order are exactly the
// increasing triples (quadruples) of the undirected graph, each once.  Any
// acyclic orientation lists each of them once too, so an operator may join
// the copy oriented from the lower to the higher (degree, id) and report
// every tuple in increasing order: the same bag, the same checksum.  Hub
// vertices then keep short child lists.  Used by ALFTJ (triangle, 4-clique)
// and by AMHJ TRI / FOUR.
#include "amj_ops.cuh"

#include <algorithm>

namespace amj {

__global__ void orient_check_kernel(const int32_t *__restrict__ s, const int32_t *__restrict__ d, uint64_t n,
                                    unsigned int *bad, int *maxv) {
    unsigned int b = 0;
    int m = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const int32_t u = s[i], v = d[i];
        b |= (u < 0 || u >= v) ? 1u : 0u;
        m = v > m ? v : m;
    }
    b = __reduce_or_sync(AMJ_FULL_MASK, b);
    m = __reduce_max_sync(AMJ_FULL_MASK, m);
    if ((threadIdx.x & 31) == 0) {
        if (b) atomicOr(bad, 1u);
        atomicMax(maxv, m);
    }
}

__global__ void degree_kernel(const int32_t *__restrict__ s, const int32_t *__restrict__ d, uint64_t n,
                              unsigned int *deg) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        atomicAdd(&deg[s[i]], 1u);
        atomicAdd(&deg[d[i]], 1u);
    }
}

__global__ void reorient_kernel(const int32_t *__restrict__ s, const int32_t *__restrict__ d, uint64_t n,
                                const unsigned int *__restrict__ deg, int32_t *__restrict__ ns,
                                int32_t *__restrict__ nd) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const int32_t u = s[i], v = d[i];
        const uint64_t ku = ((uint64_t)deg[u] << 32) | (uint32_t)u, kv = ((uint64_t)deg[v] << 32) | (uint32_t)v;
        ns[i] = ku < kv ? u : v;
        nd[i] = ku < kv ? v : u;
    }
}

int degree_ordered_copy(amj_ctx *ctx, const int32_t *c0, const int32_t *c1, uint64_t n, DBuf<int32_t> *ns,
                        DBuf<int32_t> *nd, bool *oriented) {
    *oriented = false;
    if (n == 0) return AMJ_OK;
    struct Probe {
        unsigned int bad;
        int maxv;
    };
    DBuf<Probe> pr;
    AMJ_TRY(pr.alloc(ctx, 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(pr.p, 0, sizeof(Probe), ctx->stream));
    const unsigned g = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->num_sms * 16);
    note_launch(ctx);
    orient_check_kernel<<<g, 256, 0, ctx->stream>>>(c0, c1, n, &pr.p->bad, &pr.p->maxv);
    AMJ_CUDA_TRY(cudaGetLastError());
    Probe h;
    AMJ_TRY(read_back(ctx, &h, pr.p, sizeof(h)));
    if (h.bad) return AMJ_OK;
    // per-vertex arrays are sized by the largest id: sparse ids keep the
    // relation's own order instead
    if ((uint64_t)h.maxv + 1 > 4 * n + (1ull << 20)) return AMJ_OK;
    DBuf<unsigned int> deg;
    AMJ_TRY(deg.alloc(ctx, (uint64_t)h.maxv + 1));
    AMJ_TRY(ns->alloc(ctx, n));
    AMJ_TRY(nd->alloc(ctx, n));
    AMJ_CUDA_TRY(cudaMemsetAsync(deg.p, 0, ((uint64_t)h.maxv + 1) * sizeof(unsigned int), ctx->stream));
    note_launch(ctx);
    degree_kernel<<<g, 256, 0, ctx->stream>>>(c0, c1, n, deg.p);
    note_launch(ctx);
    reorient_kernel<<<g, 256, 0, ctx->stream>>>(c0, c1, n, deg.p, ns->p, nd->p);
    AMJ_CUDA_TRY(cudaGetLastError());
    *oriented = true;
    return AMJ_OK;
}

// degrees counted on every stride-th edge: an estimate that keeps the order
// of the hubs (the counts that matter for the orientation) at a fraction of
// the atomics; any total order gives the same join result
// The counts of ids below DEG_SMEM_IDS (where generators and real graphs put
// their hubs first: R-MAT's low ids) gather in shared memory per block and
// reach the global array once per block, so a hub's increments do not
// serialise on one global counter.
constexpr uint32_t DEG_SMEM_IDS = 8192;

__global__ void degree_sample_kernel(const int32_t *__restrict__ s, const int32_t *__restrict__ d, uint64_t n,
                                     uint32_t stride, uint64_t nv, unsigned int *deg) {
    __shared__ unsigned int h[DEG_SMEM_IDS];
    for (uint32_t i = threadIdx.x; i < DEG_SMEM_IDS; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint64_t m = (n + stride - 1) / stride;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = (uint32_t)s[i * stride], b = (uint32_t)d[i * stride];
        if (a < DEG_SMEM_IDS) atomicAdd(&h[a], 1u);
        else atomicAdd(&deg[a], 1u);
        if (b < DEG_SMEM_IDS) atomicAdd(&h[b], 1u);
        else atomicAdd(&deg[b], 1u);
    }
    __syncthreads();
    const uint32_t top = nv < DEG_SMEM_IDS ? (uint32_t)nv : DEG_SMEM_IDS;
    for (uint32_t i = threadIdx.x; i < top; i += blockDim.x)
        if (h[i]) atomicAdd(&deg[i], h[i]);
}

// ---- ranks by counting over degree bins ----
// Any total order of the vertices gives the same join; it only has to put the
// hubs last.  So the vertices are not sorted by (degree, id) but counted into
// bins: one a degree below 1024, and above it 32 bins a power of two (the
// degrees of a bin differ by at most 1/32).  The order within a bin is that of
// the blocks' claims.  Two launches and no host read; sorting the degree bits
// with the largest degree read back first took eleven launches (C2, 1M
// vertices: 27 us, before 130 us).
constexpr uint32_t RANK_LINEAR = 1024;
constexpr uint32_t RANK_BINS = RANK_LINEAR + 22 * 32;
constexpr int RANK_THREADS = 1024;

__device__ __forceinline__ uint32_t degree_bin(uint32_t d) {
    if (d < RANK_LINEAR) return d;
    const uint32_t e = 31 - __clz(d);   // 10..31
    return RANK_LINEAR + (e - 10) * 32 + ((d >> (e - 5)) & 31);
}

// h += the bins of vertices [lo, hi), one shared-memory atomic a bin and warp
// (most vertices share the lowest bins)
__device__ __forceinline__ void count_bins(const unsigned int *__restrict__ deg, uint64_t lo, uint64_t hi, uint32_t *h) {
    for (uint32_t b = threadIdx.x; b < RANK_BINS; b += RANK_THREADS) h[b] = 0;
    __syncthreads();
    for (uint64_t i0 = lo + (threadIdx.x & ~31u); i0 < hi; i0 += RANK_THREADS) {
        const uint64_t i = i0 + (threadIdx.x & 31);
        const uint32_t b = i < hi ? degree_bin(deg[i]) : 0xffffffffu;
        const unsigned peers = __match_any_sync(AMJ_FULL_MASK, b);
        if (i < hi && (peers & lanemask_lt()) == 0) atomicAdd(&h[b], (uint32_t)__popc(peers));
    }
    __syncthreads();
}

__global__ __launch_bounds__(RANK_THREADS) void rank_count_kernel(const unsigned int *__restrict__ deg, uint64_t nv,
                                                                  uint64_t per, uint32_t *__restrict__ bins) {
    __shared__ uint32_t h[RANK_BINS];
    const uint64_t lo = blockIdx.x * per, hi = min(lo + per, nv);
    count_bins(deg, lo, hi, h);
    for (uint32_t b = threadIdx.x; b < RANK_BINS; b += RANK_THREADS)
        if (h[b]) atomicAdd(&bins[b], h[b]);
}

// bins: the counts of all vertices; fill: zeros.  rank[id] and inv[rank]
__global__ __launch_bounds__(RANK_THREADS) void rank_assign_kernel(const unsigned int *__restrict__ deg, uint64_t nv,
                                                                   uint64_t per, const uint32_t *__restrict__ bins,
                                                                   uint32_t *__restrict__ fill, int32_t *__restrict__ rank,
                                                                   int32_t *__restrict__ inv) {
    __shared__ uint32_t h[RANK_BINS];
    __shared__ uint32_t wsum[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t lo = blockIdx.x * per, hi = min(lo + per, nv);
    count_bins(deg, lo, hi, h);
    // h[b] = first rank of this block's vertices of bin b: the bins before it
    // (each thread two neighbouring bins) and what other blocks claimed
    const uint32_t b0 = 2 * threadIdx.x;
    const uint32_t c0 = b0 < RANK_BINS ? bins[b0] : 0u, c1 = b0 + 1 < RANK_BINS ? bins[b0 + 1] : 0u;
    const uint32_t incl = warp_inclusive_scan(c0 + c1, lane);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = wsum[lane], wi = warp_inclusive_scan(w, lane);
        wsum[lane] = wi - w;
    }
    __syncthreads();
    uint32_t at = wsum[warp] + incl - c0 - c1;
    if (b0 < RANK_BINS && h[b0]) h[b0] = at + atomicAdd(&fill[b0], h[b0]);
    at += c0;
    if (b0 + 1 < RANK_BINS && h[b0 + 1]) h[b0 + 1] = at + atomicAdd(&fill[b0 + 1], h[b0 + 1]);
    __syncthreads();
    for (uint64_t i0 = lo + (threadIdx.x & ~31u); i0 < hi; i0 += RANK_THREADS) {
        const uint64_t i = i0 + lane;
        const uint32_t b = i < hi ? degree_bin(deg[i]) : 0xffffffffu;
        const unsigned peers = __match_any_sync(AMJ_FULL_MASK, b);
        const int leader = __ffs(peers) - 1;
        uint32_t r = 0;
        if (i < hi && lane == leader) r = atomicAdd(&h[b], (uint32_t)__popc(peers));
        r = __shfl_sync(AMJ_FULL_MASK, r, leader) + __popc(peers & lanemask_lt());
        if (i < hi) {
            rank[i] = (int32_t)r;
            inv[r] = (int32_t)i;
        }
    }
}
static_assert(RANK_BINS <= 2 * RANK_THREADS, "a thread takes two bins");

int degree_ranks(amj_ctx *ctx, const int32_t *c0, const int32_t *c1, uint64_t n, DBuf<int32_t> *rank,
                 DBuf<int32_t> *inv, uint64_t *nv, bool *oriented) {
    *oriented = false;
    *nv = 0;
    if (n == 0) return AMJ_OK;
    struct Probe {
        unsigned int bad;
        int maxv;
    };
    DBuf<Probe> pr;
    AMJ_TRY(pr.alloc(ctx, 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(pr.p, 0, sizeof(Probe), ctx->stream));
    const unsigned g = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->num_sms * 16);
    note_launch(ctx);
    orient_check_kernel<<<g, 256, 0, ctx->stream>>>(c0, c1, n, &pr.p->bad, &pr.p->maxv);
    AMJ_CUDA_TRY(cudaGetLastError());
    Probe h;
    AMJ_TRY(read_back(ctx, &h, pr.p, sizeof(h)));
    if (h.bad) return AMJ_OK;
    const uint64_t V = (uint64_t)h.maxv + 1;
    // per-vertex arrays are sized by the largest id: sparse ids keep the
    // relation's own order instead
    if (V > 4 * n + (1ull << 20)) return AMJ_OK;
    if (V >= (1ull << 32)) return fail(AMJ_EUNSUPPORTED, "degree ranks: relation too large");
    // degrees, then the bins and their fill counts
    DBuf<unsigned int> deg;
    AMJ_TRY(deg.alloc(ctx, V + 2 * RANK_BINS));
    AMJ_CUDA_TRY(cudaMemsetAsync(deg.p, 0, (V + 2 * RANK_BINS) * sizeof(unsigned int), ctx->stream));
    // relations of 2^20 edges or more rank by degrees counted on every 4th edge
    const uint32_t stride = n >= (1ull << 20) ? 4u : 1u;
    note_launch(ctx);
    degree_sample_kernel<<<(unsigned)std::min<uint64_t>(g, (uint64_t)ctx->num_sms * 4), 256, 0, ctx->stream>>>(
        c0, c1, n, stride, V, deg.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    AMJ_TRY(rank->alloc(ctx, V));
    AMJ_TRY(inv->alloc(ctx, V));
    const uint64_t blocks = std::min<uint64_t>((V + RANK_THREADS - 1) / RANK_THREADS, (uint64_t)ctx->num_sms);
    const uint64_t per = (V + blocks - 1) / blocks;
    uint32_t *bins = deg.p + V;
    note_launch(ctx);
    rank_count_kernel<<<(unsigned)blocks, RANK_THREADS, 0, ctx->stream>>>(deg.p, V, per, bins);
    note_launch(ctx);
    rank_assign_kernel<<<(unsigned)blocks, RANK_THREADS, 0, ctx->stream>>>(deg.p, V, per, bins, bins + RANK_BINS,
                                                                          rank->p, inv->p);
    AMJ_CUDA_TRY(cudaGetLastError());
    *nv = V;
    *oriented = true;
    return AMJ_OK;
}

}  // namespace amj
