// IndexedTrie construction and .tr (de)serialisation for 2-column relations.
//
// Reference: constructSortedTrie (LFTJ-GPU/multi_partitioning.cuh:129-293)
// sorts the tuples with CUB / Thrust, marks value changes (extractMasks,
// :104), and compacts the distinct values and their child offsets with
// segmented selects and scans.  Here: one min/max reduction sizes a compact
// sort key (c0 - min0) << bits1 | (c1 - min1) so the LSD radix sort runs only
// over the bits that vary (40 bits -> 5 passes for 2^20 vertices), then one
// kernel unpacks level 1 and flags group heads, a scan numbers the heads and
// a scatter writes level 0 and its offsets.  A dense row-pointer array over
// the level-0 value range is added when that range is small, so a probe can
// find a value's children with one load instead of a binary search.
#include "amj_ops.cuh"

#include <cstdio>
#include <cstring>
#include <vector>

namespace amj {

__global__ void minmax_pairs_kernel(const int32_t *__restrict__ c0, const int32_t *__restrict__ c1, uint64_t n,
                                    uint32_t *mm /* min0,max0,min1,max1 in sign-flipped order */) {
    uint32_t mn0 = 0xffffffffu, mx0 = 0, mn1 = 0xffffffffu, mx1 = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t a = (uint32_t)c0[i] ^ 0x80000000u, b = (uint32_t)c1[i] ^ 0x80000000u;
        mn0 = min(mn0, a); mx0 = max(mx0, a);
        mn1 = min(mn1, b); mx1 = max(mx1, b);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        mn0 = min(mn0, __shfl_xor_sync(AMJ_FULL_MASK, mn0, d));
        mx0 = max(mx0, __shfl_xor_sync(AMJ_FULL_MASK, mx0, d));
        mn1 = min(mn1, __shfl_xor_sync(AMJ_FULL_MASK, mn1, d));
        mx1 = max(mx1, __shfl_xor_sync(AMJ_FULL_MASK, mx1, d));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&mm[0], mn0); atomicMax(&mm[1], mx0);
        atomicMin(&mm[2], mn1); atomicMax(&mm[3], mx1);
    }
}

__global__ void pack_trie_keys_kernel(const int32_t *__restrict__ c0, const int32_t *__restrict__ c1, uint64_t n,
                                      uint32_t min0, uint32_t min1, int bits1, uint64_t *__restrict__ items) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t a = ((uint32_t)c0[i] ^ 0x80000000u) - min0;
        uint64_t b = ((uint32_t)c1[i] ^ 0x80000000u) - min1;
        items[i] = (a << bits1) | b;
    }
}

__device__ __forceinline__ int32_t unflip(uint64_t v, uint32_t mn) {
    return (int32_t)(((uint32_t)v + mn) ^ 0x80000000u);
}

__global__ void unpack_trie_kernel(const uint64_t *__restrict__ items, uint64_t n, uint32_t min0, uint32_t min1,
                                   int bits1, int32_t *__restrict__ data1, int32_t *__restrict__ src1,
                                   uint32_t *__restrict__ head) {
    const uint64_t m1 = bits1 >= 64 ? ~0ull : ((1ull << bits1) - 1);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = items[i];
        data1[i] = unflip(v & m1, min1);
        src1[i] = unflip(v >> bits1, min0);
        head[i] = (i == 0 || (items[i - 1] >> bits1) != (v >> bits1)) ? 1u : 0u;
    }
}

__global__ void scatter_level0_kernel(const uint64_t *__restrict__ items, const uint32_t *__restrict__ head,
                                      const uint32_t *__restrict__ pos, uint64_t n, uint32_t min0, int bits1,
                                      int32_t *__restrict__ data0, uint64_t *__restrict__ off0, uint64_t len0) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        // head[] was scanned in place into pos[]; recompute the head flag
        const bool h = (i == 0) || ((items[i - 1] >> bits1) != (items[i] >> bits1));
        if (h) {
            const uint32_t p = pos[i];
            data0[p] = unflip(items[i] >> bits1, min0);
            off0[p] = i;
        }
        if (i == 0) off0[len0] = n;
    }
    (void)head;
}

// adjacent equal items of a sorted array (duplicate rows), counted per block
__global__ void count_dups_kernel(const uint64_t *__restrict__ items, uint64_t n, unsigned long long *dups) {
    unsigned long long c = 0;
    for (uint64_t i = 1 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c += items[i] == items[i - 1];
    c = warp_sum(c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(dups, c);
}

__global__ void first_of_run_kernel(const uint64_t *__restrict__ items, uint64_t n, uint32_t *__restrict__ flag) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        flag[i] = (i == 0 || items[i] != items[i - 1]) ? 1u : 0u;
}

__global__ void compact_runs_kernel(const uint64_t *__restrict__ items, const uint32_t *__restrict__ pos, uint64_t n,
                                    uint64_t *__restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (i == 0 || items[i] != items[i - 1]) out[pos[i]] = items[i];
}

// child counts of every level-0 value, indexed densely by value - min
__global__ void dense_counts_kernel(const int32_t *__restrict__ data0, const uint64_t *__restrict__ off0,
                                    uint64_t len0, int32_t vmin, uint64_t *__restrict__ counts) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < len0; i += (uint64_t)gridDim.x * blockDim.x)
        counts[(uint64_t)((int64_t)data0[i] - (int64_t)vmin)] = off0[i + 1] - off0[i];
}

static unsigned grid_for(amj_ctx *ctx, uint64_t n) {
    uint64_t g = (n + 255) / 256, cap = (uint64_t)ctx->num_sms * 16;
    return (unsigned)(g == 0 ? 1 : (g > cap ? cap : g));
}

static int bits_for(uint32_t range) {
    int b = 0;
    while (b < 32 && (range >> b) != 0) b++;
    return b;
}

int build_trie2(amj_ctx *ctx, const int32_t *d_c0, const int32_t *d_c1, uint64_t n, Trie2 *out, bool distinct,
                int32_t vmax, const uint32_t *mm_known) {
    if (n >= (1ull << 32) - 4096) return fail(AMJ_EUNSUPPORTED, "trie build: 2^32 or more rows");
    out->len1 = n;
    if (n == 0) {
        out->len0 = 0;
        AMJ_TRY(out->off0.alloc(ctx, 1));
        AMJ_CUDA_TRY(cudaMemsetAsync(out->off0.p, 0, sizeof(uint64_t), ctx->stream));
        AMJ_TRY(out->data0.alloc(ctx, 1));
        AMJ_TRY(out->data1.alloc(ctx, TRIE_LEVEL1_PAD));
        return AMJ_OK;
    }
    uint32_t h_mm[4];   // flipped min / max of both columns
    if (mm_known) {
        std::memcpy(h_mm, mm_known, sizeof(h_mm));
    } else if (vmax >= 0) {
        // the caller knows every value lies in [0, vmax]
        h_mm[0] = h_mm[2] = 0x80000000u;
        h_mm[1] = h_mm[3] = (uint32_t)vmax ^ 0x80000000u;
    } else {
        DBuf<uint32_t> mm;
        AMJ_TRY(mm.alloc(ctx, 8));
        const uint32_t init[4] = {0xffffffffu, 0u, 0xffffffffu, 0u};
        AMJ_CUDA_TRY(cudaMemcpyAsync(mm.p, init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
        note_launch(ctx);
        minmax_pairs_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(d_c0, d_c1, n, mm.p);
        AMJ_CUDA_TRY(cudaGetLastError());
        AMJ_CUDA_TRY(cudaMemcpyAsync(h_mm, mm.p, sizeof(h_mm), cudaMemcpyDeviceToHost, ctx->stream));
        AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    }
    const uint32_t min0 = h_mm[0], min1 = h_mm[2];
    const int bits0 = bits_for(h_mm[1] - min0), bits1 = bits_for(h_mm[3] - min1);
    out->range1 = (uint64_t)(h_mm[3] - min1) + 1;

    DBuf<uint64_t> a, b;
    AMJ_TRY(a.alloc(ctx, n));
    AMJ_TRY(b.alloc(ctx, n));
    note_launch(ctx);
    pack_trie_keys_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(d_c0, d_c1, n, min0, min1, bits1, a.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    uint64_t *sorted = nullptr;
    AMJ_TRY(radix_sort_u64(ctx, a.p, b.p, n, SK_IDENT, 0, bits0 + bits1, &sorted));
    // set semantics (distinct): repeated rows are adjacent after the sort;
    // they are counted beside the level-1 unpack and, when there are some,
    // dropped and the unpack redone
    DBuf<unsigned long long> dups;
    if (distinct && n > 1) {
        AMJ_TRY(dups.alloc(ctx, 1));
        AMJ_CUDA_TRY(cudaMemsetAsync(dups.p, 0, sizeof(unsigned long long), ctx->stream));
        note_launch(ctx);
        count_dups_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sorted, n, dups.p);
        AMJ_CUDA_TRY(cudaGetLastError());
    }
    AMJ_TRY(out->data1.alloc(ctx, n + TRIE_LEVEL1_PAD));
    AMJ_TRY(out->src1.alloc(ctx, n));
    DBuf<uint32_t> head;
    AMJ_TRY(head.alloc(ctx, n + 1));
    uint32_t len0 = 0;
    unsigned long long h_dups = 0;
    for (int round = 0; round < 2; round++) {
        note_launch(ctx);
        unpack_trie_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sorted, n, min0, min1, bits1, out->data1.p,
                                                                       out->src1.p, head.p);
        AMJ_CUDA_TRY(cudaGetLastError());
        AMJ_TRY(scan_exclusive_u32(ctx, head.p, head.p, n, head.p + n));
        AMJ_CUDA_TRY(cudaMemcpyAsync(&len0, head.p + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
        if (round == 0 && dups.p)
            AMJ_CUDA_TRY(cudaMemcpyAsync(&h_dups, dups.p, sizeof(h_dups), cudaMemcpyDeviceToHost, ctx->stream));
        AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        if (round > 0 || h_dups == 0) break;
        DBuf<uint32_t> pos;
        AMJ_TRY(pos.alloc(ctx, n));
        note_launch(ctx);
        first_of_run_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sorted, n, pos.p);
        AMJ_CUDA_TRY(cudaGetLastError());
        AMJ_TRY(scan_exclusive_u32(ctx, pos.p, pos.p, n, nullptr));
        uint64_t *other = sorted == a.p ? b.p : a.p;
        note_launch(ctx);
        compact_runs_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sorted, pos.p, n, other);
        AMJ_CUDA_TRY(cudaGetLastError());
        sorted = other;
        n -= h_dups;
        out->len1 = n;
    }
    out->len0 = len0;
    AMJ_TRY(out->data0.alloc(ctx, len0));
    AMJ_TRY(out->off0.alloc(ctx, (uint64_t)len0 + 1));
    note_launch(ctx);
    scatter_level0_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sorted, head.p, head.p, n, min0, bits1,
                                                                      out->data0.p, out->off0.p, len0);
    AMJ_CUDA_TRY(cudaGetLastError());
    // dense row pointers when the level-0 value range is small against the trie
    const uint64_t range = (uint64_t)(h_mm[1] - min0) + 1;
    if (range <= 4 * (uint64_t)len0 + 4096 && range < (1ull << 31)) {
        out->rp_min = (int32_t)(min0 ^ 0x80000000u);
        out->rp_count = range;
        AMJ_TRY(out->rowptr.alloc(ctx, range + 1));
        AMJ_CUDA_TRY(cudaMemsetAsync(out->rowptr.p, 0, (range + 1) * sizeof(uint64_t), ctx->stream));
        note_launch(ctx);
        dense_counts_kernel<<<grid_for(ctx, len0), 256, 0, ctx->stream>>>(out->data0.p, out->off0.p, len0,
                                                                          out->rp_min, out->rowptr.p);
        AMJ_CUDA_TRY(cudaGetLastError());
        AMJ_TRY(scan_exclusive_u64(ctx, out->rowptr.p, out->rowptr.p, range + 1, nullptr));
    }
    return AMJ_OK;
}

// ---- 2-level tries of a degree-ranked copy: rows by counting ----
// Every value lies in [0, nv) and every row's first value is below its
// second, so the rows can be bucketed by their first value directly: one pass
// ranks the edges, counts them per value and keeps each edge's place in its
// row, a scan gives the row starts, one pass writes the second values to start
// + place, then each row is sorted on its own.  Level 0 lists every rank, so
// nothing is compacted and one host read (repeated rows, longest row) ends the
// build: 26 device operations and 3 host reads a triangle query of 64K edges
// instead of 49 and 6 (435 to 276 us), 1.42 instead of 1.80 ms of builds on C2.
// After the degree
// ranking a row holds the higher-ranked neighbours of one vertex, at most
// sqrt(2 n) of them, and most rows hold a few: a warp sorts a row of up to
// RK_WARP_MAX values in registers (a bitonic network over shuffles); a block
// sorts the longer rows, up to RK_BLOCK_MAX, in shared memory.  A graph with a longer row takes the radix-sort build.
// Repeated rows (adjacent after the sort) are dropped by a compaction pass
// when there are any.
constexpr uint32_t RK_WARP_MAX = 1024;
constexpr uint32_t RK_BLOCK_MAX = 32768;   // 132 KB of shared memory, padded
constexpr int RK_SORT_WARPS = 8;

// Ranked edges (the lower rank first), the count of every lower rank, each
// edge's place among those of its lower rank (the value its atomic returned),
// and the longest row.  Four edges a thread, so that the dependent lookups of
// one overlap those of the others.
__global__ __launch_bounds__(256) void rk_edges_kernel(const int32_t *__restrict__ s, const int32_t *__restrict__ d,
                                                       uint64_t n, const int32_t *__restrict__ rank,
                                                       uint32_t *__restrict__ cnt, int32_t *__restrict__ lo,
                                                       int32_t *__restrict__ hi, uint32_t *__restrict__ place,
                                                       unsigned int *__restrict__ longest) {
    const uint64_t i0 = blockIdx.x * 1024ull + threadIdx.x;
    int32_t u[4], v[4];
    uint32_t p[4], m = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint64_t i = i0 + k * 256;
        if (i < n) {
            u[k] = rank[s[i]];
            v[k] = rank[d[i]];
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (i0 + k * 256 < n) p[k] = atomicAdd(&cnt[min(u[k], v[k])], 1u);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint64_t i = i0 + k * 256;
        if (i < n) {
            lo[i] = min(u[k], v[k]);
            hi[i] = max(u[k], v[k]);
            place[i] = p[k];
            m = max(m, p[k] + 1);
        }
    }
    m = __reduce_max_sync(AMJ_FULL_MASK, m);
    if ((threadIdx.x & 31) == 0 && m > ld_volatile_u32(longest)) atomicMax(longest, m);
}

__global__ __launch_bounds__(256) void rk_scatter_kernel(const int32_t *__restrict__ lo, const int32_t *__restrict__ hi,
                                                         const uint32_t *__restrict__ place, uint64_t n,
                                                         const uint32_t *__restrict__ start,
                                                         int32_t *__restrict__ data1) {
    const uint64_t i0 = blockIdx.x * 1024ull + threadIdx.x;
    uint32_t p[4];
    int32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint64_t i = i0 + k * 256;
        if (i < n) {
            p[k] = start[lo[i]] + place[i];
            v[k] = hi[i];
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (i0 + k * 256 < n) data1[p[k]] = v[k];
}

// row v = data1[s, s + len), 32 (E / 2) < len <= 32 E: sorted in place, its
// level-0 value into src1, its number of distinct values into uniq[v]
template <int E>
__device__ __forceinline__ uint32_t rk_warp_row(int32_t *__restrict__ data1, int32_t *__restrict__ src1,
                                            uint32_t *__restrict__ uniq, uint32_t s, uint32_t len, uint64_t v,
                                            int32_t value, uint32_t lane) {
    int32_t x[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const uint32_t i = e * 32u + lane;   // coalesced loads; the network fixes the order
        x[e] = i < len ? data1[s + i] : INT32_MAX;
    }
    warp_bitonic_sort<E>(x, lane);
    const int32_t prev = __shfl_up_sync(AMJ_FULL_MASK, x[E - 1], 1);
    uint32_t u = 0;
#pragma unroll
    for (int e = 0; e < E; e++) {
        const uint32_t i = lane * E + e;
        if (i < len) {
            const int32_t before = e ? x[e - 1] : prev;
            u += (i == 0 || x[e] != before) ? 1u : 0u;
            data1[s + i] = x[e];
            src1[s + i] = value;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) u += __shfl_xor_sync(AMJ_FULL_MASK, u, d);
    if (lane == 0) uniq[v] = u;
    return u;
}

// The rows of one trie, or of several end to end: distinct values are counted for
// each trie.  row[p] is the first row of trie p > 0.
struct RowParts {
    uint32_t row[TRIE_JOBS_MAX] = {0, 0xffffffffu, 0xffffffffu};
    __device__ __forceinline__ int of(uint64_t v) const { return (v >= row[1] ? 1 : 0) + (v >= row[2] ? 1 : 0); }
};
static_assert(TRIE_JOBS_MAX == 3, "RowParts::of");

// One warp a row, the row's values in registers (rows of up to RK_WARP_MAX);
// longer rows are listed for the block kernel.
__global__ __launch_bounds__(RK_SORT_WARPS * 32, 4) void rk_sort_rows_kernel(const uint32_t *__restrict__ start,
                                                                           const int32_t *__restrict__ values,
                                                                           uint64_t nv, int32_t *__restrict__ data1,
                                                                           int32_t *__restrict__ src1,
                                                                           uint32_t *__restrict__ uniq,
                                                                           uint32_t *__restrict__ longs,
                                                                           unsigned int *__restrict__ nlong,
                                                                           const RowParts parts,
                                                                           unsigned long long *__restrict__ distinct) {
    __shared__ uint32_t usum[TRIE_JOBS_MAX];
    if (threadIdx.x < TRIE_JOBS_MAX) usum[threadIdx.x] = 0;
    __syncthreads();
    uint32_t u = 0;   // distinct values of this warp's rows of the current part
    int part = 0;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t warps = (uint64_t)gridDim.x * RK_SORT_WARPS;
    for (uint64_t v = blockIdx.x * (uint64_t)RK_SORT_WARPS + w; v < nv; v += warps) {
        const uint32_t s = start[v], len = start[v + 1] - s;
        const int32_t value = values ? values[v] : (int32_t)v;
        const int p = parts.of(v);
        if (p != part) {
            if (lane == 0) atomicAdd(&usum[part], u);
            u = 0;
            part = p;
        }
        if (len <= 1) {
            if (len == 1 && lane == 0) src1[s] = value;
            if (lane == 0) uniq[v] = len;
            u += len;
        } else if (len <= 32) {
            u += rk_warp_row<1>(data1, src1, uniq, s, len, v, value, lane);
        } else if (len <= 64) {
            u += rk_warp_row<2>(data1, src1, uniq, s, len, v, value, lane);
        } else if (len <= 128) {
            u += rk_warp_row<4>(data1, src1, uniq, s, len, v, value, lane);
        } else if (len <= 256) {
            u += rk_warp_row<8>(data1, src1, uniq, s, len, v, value, lane);
        } else if (len <= 512) {
            u += rk_warp_row<16>(data1, src1, uniq, s, len, v, value, lane);
        } else if (len <= RK_WARP_MAX) {
            u += rk_warp_row<32>(data1, src1, uniq, s, len, v, value, lane);
        } else if (lane == 0) {
            longs[atomicAdd(nlong, 1u)] = (uint32_t)v;
            uniq[v] = 0;
        }
    }
    if (lane == 0) atomicAdd(&usum[part], u);
    __syncthreads();
    if (threadIdx.x < TRIE_JOBS_MAX && usum[threadIdx.x])
        atomicAdd(&distinct[threadIdx.x], (unsigned long long)usum[threadIdx.x]);
}

// A row of up to 1024 E values sorted by a block of 1024 threads in shared
// memory: E warps sort 1024 values each in registers, then the runs are merged
// pairwise, each thread placing E consecutive values of the result (its start
// in the two runs by the merge path's binary search).  Values sit one word in
// 33 apart, so that a lane's consecutive values fall in different banks.  (A
// bitonic network over shared memory took 316 us for the long rows of three
// 1M-edge R-MAT relations, this 76 us.)
__device__ __forceinline__ uint32_t rk_pad(uint32_t i) { return i + (i >> 5); }

template <int E>
__device__ __forceinline__ void rk_block_sort(int32_t *x, const int32_t *__restrict__ row, uint32_t len) {
    const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (w < E) {
        int32_t v[32];
#pragma unroll
        for (int e = 0; e < 32; e++) {
            const uint32_t i = w * 1024 + e * 32 + lane;
            v[e] = i < len ? row[i] : INT32_MAX;
        }
        warp_bitonic_sort<32>(v, lane);
#pragma unroll
        for (int e = 0; e < 32; e++) x[rk_pad(w * 1024 + lane * 32 + e)] = v[e];
    }
    __syncthreads();
    for (uint32_t width = 1024; width < 1024u * E; width *= 2) {
        const uint32_t out0 = t * E, base = out0 / (2 * width) * (2 * width), diag = out0 - base;
        const uint32_t A = base, B = base + width;
        uint32_t lo = diag > width ? diag - width : 0, hi = min(diag, width);
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (x[rk_pad(A + mid)] <= x[rk_pad(B + diag - 1 - mid)]) lo = mid + 1;
            else hi = mid;
        }
        uint32_t i = lo, j = diag - lo;
        int32_t v[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const bool a = j >= width || (i < width && x[rk_pad(A + i)] <= x[rk_pad(B + j)]);
            v[e] = a ? x[rk_pad(A + i)] : x[rk_pad(B + j)];
            i += a ? 1u : 0u;
            j += a ? 0u : 1u;
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) x[rk_pad(out0 + e)] = v[e];
        __syncthreads();
    }
}

// One block a listed row (RK_WARP_MAX < length <= RK_BLOCK_MAX); the blocks
// take the list's rows in turn
__global__ __launch_bounds__(1024) void rk_sort_long_kernel(const uint32_t *__restrict__ start,
                                                            const int32_t *__restrict__ values,
                                                            int32_t *__restrict__ data1, int32_t *__restrict__ src1,
                                                            uint32_t *__restrict__ uniq,
                                                            const uint32_t *__restrict__ longs,
                                                            const unsigned int *__restrict__ nlong,
                                                            const RowParts parts,
                                                            unsigned long long *__restrict__ distinct) {
    extern __shared__ int32_t x[];   // RK_BLOCK_MAX values, padded
    __shared__ uint32_t usum;
    const uint32_t t = threadIdx.x, nt = blockDim.x;
    for (uint32_t r = blockIdx.x; r < *nlong; r += gridDim.x) {
        const uint32_t v = longs[r], s = start[v], len = start[v + 1] - s;
        if (len > RK_BLOCK_MAX) continue;   // the host takes the radix build
        if (t == 0) usum = 0;
        if (len <= 2048) rk_block_sort<2>(x, data1 + s, len);
        else if (len <= 4096) rk_block_sort<4>(x, data1 + s, len);
        else if (len <= 8192) rk_block_sort<8>(x, data1 + s, len);
        else if (len <= 16384) rk_block_sort<16>(x, data1 + s, len);
        else rk_block_sort<32>(x, data1 + s, len);
        const int32_t value = values ? values[v] : (int32_t)v;
        uint32_t u = 0;
        for (uint32_t i = t; i < len; i += nt) {
            const int32_t y = x[rk_pad(i)];
            u += (i == 0 || y != x[rk_pad(i - 1)]) ? 1u : 0u;
            data1[s + i] = y;
            src1[s + i] = value;
        }
        u = warp_sum(u);
        if ((t & 31) == 0 && u) atomicAdd(&usum, u);
        __syncthreads();
        if (t == 0) {
            uniq[v] = usum;
            atomicAdd(&distinct[parts.of(v)], (unsigned long long)usum);
        }
        __syncthreads();
    }
}

static int launch_sort_long(amj_ctx *ctx, const uint32_t *start, const int32_t *values, int32_t *data1, int32_t *src1,
                            uint32_t *uniq, const uint32_t *longs, const unsigned int *nlong, const RowParts &parts,
                            unsigned long long *distinct) {
    constexpr size_t smem = (RK_BLOCK_MAX + RK_BLOCK_MAX / 32) * sizeof(int32_t);
    AMJ_CUDA_TRY(cudaFuncSetAttribute(rk_sort_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    note_launch(ctx);
    rk_sort_long_kernel<<<ctx->num_sms, 1024, smem, ctx->stream>>>(start, values, data1, src1, uniq, longs, nlong,
                                                                   parts, distinct);
    AMJ_CUDA_TRY(cudaGetLastError());
    return AMJ_OK;
}

// repeated rows present: row v's distinct values move to ustart[v] (a warp a row)
__global__ void rk_compact_kernel(const uint32_t *__restrict__ start, const uint32_t *__restrict__ ustart,
                                  const int32_t *__restrict__ values, uint64_t nv,
                                  const int32_t *__restrict__ data1, int32_t *__restrict__ out1,
                                  int32_t *__restrict__ outsrc) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv; v += warps) {
        const uint32_t s = start[v], len = start[v + 1] - s;
        uint32_t at = ustart[v];
        for (uint32_t i0 = 0; i0 < len; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool keep = i < len && (i == 0 || data1[s + i] != data1[s + i - 1]);
            const unsigned b = __ballot_sync(AMJ_FULL_MASK, keep);
            if (keep) {
                const uint32_t o = at + __popc(b & ((1u << lane) - 1u));
                out1[o] = data1[s + i];
                outsrc[o] = values ? values[v] : (int32_t)v;
            }
            at += __popc(b);
        }
    }
}

// level 0 (every rank) and the row pointers
__global__ void rk_level0_kernel(const uint32_t *__restrict__ start, uint64_t nv, int32_t *__restrict__ data0,
                                 uint64_t *__restrict__ rowptr) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v <= nv; v += (uint64_t)gridDim.x * blockDim.x) {
        rowptr[v] = start[v];
        if (v < nv) data0[v] = (int32_t)v;
    }
}

int build_trie2_ranked(amj_ctx *ctx, const int32_t *d_c0, const int32_t *d_c1, uint64_t n, const int32_t *rank,
                       uint64_t nv, Trie2 *out) {
    if (n == 0 || nv == 0) return build_trie2(ctx, d_c0, d_c1, n, out, true, -1);
    // ranked edges with their places in their rows; a scan of the counts
    DBuf<int32_t> lo, hi;
    DBuf<uint32_t> start, place;
    struct Ctr {
        unsigned int longest, nlong;   // longest row; rows listed for the block kernel
        unsigned long long distinct[TRIE_JOBS_MAX];
    };
    const RowParts one;
    AMJ_TRY(lo.alloc(ctx, n));
    AMJ_TRY(hi.alloc(ctx, n));
    AMJ_TRY(place.alloc(ctx, n));
    // row starts, then the counters (8-byte aligned)
    const uint64_t ctr_at = (nv + 2) / 2 * 2;
    AMJ_TRY(start.alloc(ctx, ctr_at + sizeof(Ctr) / sizeof(uint32_t)));
    Ctr *ctr = reinterpret_cast<Ctr *>(start.p + ctr_at);
    AMJ_CUDA_TRY(cudaMemsetAsync(start.p, 0, ctr_at * sizeof(uint32_t) + sizeof(Ctr), ctx->stream));
    const uint64_t tiles = (n + 1023) / 1024;
    note_launch(ctx);
    rk_edges_kernel<<<(unsigned)tiles, 256, 0, ctx->stream>>>(d_c0, d_c1, n, rank, start.p, lo.p, hi.p, place.p,
                                                              &ctr->longest);
    AMJ_CUDA_TRY(cudaGetLastError());
    if (nv >= (1ull << 31) || n >= (1ull << 32) - 4096)
        return build_trie2(ctx, lo.p, hi.p, n, out, true, (int32_t)(nv - 1));
    AMJ_TRY(scan_exclusive_u32(ctx, start.p, start.p, nv + 1, nullptr));
    // the rows, each sorted, with their distinct counts
    AMJ_TRY(out->data1.alloc(ctx, n + TRIE_LEVEL1_PAD));
    AMJ_TRY(out->src1.alloc(ctx, n));
    DBuf<uint32_t> uniq, longs;
    AMJ_TRY(uniq.alloc(ctx, nv + 1));
    AMJ_TRY(longs.alloc(ctx, std::max<uint64_t>(1, n / (RK_WARP_MAX + 1) + 1)));
    note_launch(ctx);
    rk_scatter_kernel<<<(unsigned)tiles, 256, 0, ctx->stream>>>(lo.p, hi.p, place.p, n, start.p, out->data1.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    const unsigned gs = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((nv + RK_SORT_WARPS - 1) / RK_SORT_WARPS,
                                                                           (uint64_t)ctx->num_sms * 8));
    note_launch(ctx);
    rk_sort_rows_kernel<<<gs, RK_SORT_WARPS * 32, 0, ctx->stream>>>(start.p, nullptr, nv, out->data1.p, out->src1.p, uniq.p,
                                                                    longs.p, &ctr->nlong, one, ctr->distinct);
    AMJ_CUDA_TRY(cudaGetLastError());
    // in rank order a row holds about sqrt(2 n) values at most unless edges
    // repeat: small relations launch the block sort only when they turn out to
    // need it
    const bool long_rows = n >= (1u << 18);
    if (long_rows) {
        AMJ_TRY(launch_sort_long(ctx, start.p, nullptr, out->data1.p, out->src1.p, uniq.p, longs.p, &ctr->nlong,
                                 one, ctr->distinct));
    }
    // level 0 and the row pointers, unless rows repeat or are too long
    out->len0 = nv;
    out->rp_min = 0;
    out->rp_count = nv;
    AMJ_TRY(out->data0.alloc(ctx, nv));
    AMJ_TRY(out->rowptr.alloc(ctx, nv + 1));
    out->off0.release();
    out->off0.ctx = nullptr;   // a view: the row pointers of every rank
    out->off0.p = out->rowptr.p;
    out->off0.n = nv + 1;
    note_launch(ctx);
    rk_level0_kernel<<<grid_for(ctx, nv + 1), 256, 0, ctx->stream>>>(start.p, nv, out->data0.p, out->rowptr.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    Ctr h{};
    AMJ_TRY(read_back(ctx, &h, ctr, sizeof(h)));
    if (!long_rows && h.nlong && h.longest <= RK_BLOCK_MAX) {
        AMJ_TRY(launch_sort_long(ctx, start.p, nullptr, out->data1.p, out->src1.p, uniq.p, longs.p, &ctr->nlong,
                                 one, ctr->distinct));
        AMJ_TRY(read_back(ctx, &h, ctr, sizeof(h)));
    }
    if (h.longest > RK_BLOCK_MAX) {
        *out = Trie2();
        return build_trie2(ctx, lo.p, hi.p, n, out, true, (int32_t)(nv - 1));
    }
    out->len1 = h.distinct[0];
    if (h.distinct[0] == n) return AMJ_OK;
    // repeated rows: the distinct values of every row, compacted
    AMJ_CUDA_TRY(cudaMemsetAsync(uniq.p + nv, 0, sizeof(uint32_t), ctx->stream));
    AMJ_TRY(scan_exclusive_u32(ctx, uniq.p, uniq.p, nv + 1, nullptr));
    DBuf<int32_t> d1, s1;
    AMJ_TRY(d1.alloc(ctx, h.distinct[0] + TRIE_LEVEL1_PAD));
    AMJ_TRY(s1.alloc(ctx, h.distinct[0] ? h.distinct[0] : 1));
    note_launch(ctx);
    rk_compact_kernel<<<grid_for(ctx, nv * 32), 256, 0, ctx->stream>>>(start.p, uniq.p, nullptr, nv, out->data1.p, d1.p,
                                                                       s1.p);
    note_launch(ctx);
    rk_level0_kernel<<<grid_for(ctx, nv + 1), 256, 0, ctx->stream>>>(uniq.p, nv, out->data0.p, out->rowptr.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    out->data1 = std::move(d1);
    out->src1 = std::move(s1);
    return AMJ_OK;
}

// ---- 2-level tries of several relations, rows by counting ----
// The tries of a triangle query's relations, built together as the ranked trie
// is: counts per first-column value with each row's place, one scan, one move,
// one sort of all rows, so that the query has ten launches and two host reads
// for its builds instead of some hundred and nine (three relations of 1M edges:
// 1.03 ms one by one, 0.36 ms together).  Level 0 lists every
// value of the first column's range, which has to be dense (at most 4 n + 4096
// values).  Repeated rows are dropped by a compaction of the relations that have
// some (1.05 to 1.41 ms with one repeated row in each of three 1M-edge relations; 2.11 ms
// when one sent all of them to the radix sort).  A relation with a wider range, or with a row above
// RK_BLOCK_MAX, is built alone.
struct TrieJob {
    const int32_t *c0, *c1;
    uint32_t n, nrows;   // edges; values of the first column's range
    uint32_t row0, e0;   // first row and first edge in the shared arrays
    uint32_t min0;       // least first value (sign flipped)
    uint64_t *rowptr;
};
struct TrieJobs {
    TrieJob j[TRIE_JOBS_MAX];
};

// least and greatest value of both columns: mm[0..3] of a relation = ~min0, max0,
// ~min1, max1, sign flipped (zeros are neutral); one set of atomics a block
__global__ __launch_bounds__(256) void tries_minmax_kernel(const __grid_constant__ TrieJobs A,
                                                           uint32_t *__restrict__ mm) {
    const TrieJob &J = A.j[blockIdx.y];
    uint32_t m[4] = {0, 0, 0, 0};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < J.n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = (uint32_t)J.c0[i] ^ 0x80000000u, b = (uint32_t)J.c1[i] ^ 0x80000000u;
        m[0] = max(m[0], ~a);
        m[1] = max(m[1], a);
        m[2] = max(m[2], ~b);
        m[3] = max(m[3], b);
    }
    __shared__ uint32_t s[4][8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        m[k] = __reduce_max_sync(AMJ_FULL_MASK, m[k]);
        if ((threadIdx.x & 31) == 0) s[k][threadIdx.x >> 5] = m[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        uint32_t x = 0;
        for (int w = 0; w < 8; w++) x = max(x, s[threadIdx.x][w]);
        atomicMax(&mm[4 * blockIdx.y + threadIdx.x], x);
    }
}

// One tile of edges a block.  The first TRIES_SMEM_ROWS rows, where generators
// and real graphs put their hubs, are counted in shared memory and reach the
// global count once a block: a hub's atomics do not queue on one address (3M
// edges of three R-MAT relations: 106 us with global counts only, 37 us now).
constexpr uint32_t TRIES_SMEM_ROWS = 4096;
constexpr int TRIES_PER_THREAD = 16;

__global__ __launch_bounds__(256) void tries_count_kernel(const __grid_constant__ TrieJobs A, uint32_t *__restrict__ cnt,
                                                          uint32_t *__restrict__ place) {
    __shared__ uint32_t h[TRIES_SMEM_ROWS];
    const TrieJob &J = A.j[blockIdx.y];
    const uint32_t i0 = blockIdx.x * (256u * TRIES_PER_THREAD);
    if (i0 >= J.n) return;
    for (uint32_t i = threadIdx.x; i < TRIES_SMEM_ROWS; i += 256) h[i] = 0;
    __syncthreads();
    uint32_t row[TRIES_PER_THREAD], p[TRIES_PER_THREAD];
#pragma unroll
    for (int k = 0; k < TRIES_PER_THREAD; k++) {
        const uint32_t i = i0 + k * 256 + threadIdx.x;
        row[k] = i < J.n ? ((uint32_t)J.c0[i] ^ 0x80000000u) - J.min0 : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < TRIES_PER_THREAD; k++) {
        if (row[k] < TRIES_SMEM_ROWS) p[k] = atomicAdd(&h[row[k]], 1u);
        else if (row[k] != 0xffffffffu) p[k] = atomicAdd(&cnt[J.row0 + row[k]], 1u);
    }
    __syncthreads();
    // h[row] becomes the block's first place in the row
    for (uint32_t i = threadIdx.x; i < TRIES_SMEM_ROWS; i += 256)
        if (h[i]) h[i] = atomicAdd(&cnt[J.row0 + i], h[i]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TRIES_PER_THREAD; k++)
        if (row[k] != 0xffffffffu)
            place[J.e0 + i0 + k * 256 + threadIdx.x] = p[k] + (row[k] < TRIES_SMEM_ROWS ? h[row[k]] : 0u);
}

__global__ __launch_bounds__(256) void tries_scatter_kernel(const __grid_constant__ TrieJobs A,
                                                            const uint32_t *__restrict__ start,
                                                            const uint32_t *__restrict__ place,
                                                            int32_t *__restrict__ data1) {
    const TrieJob &J = A.j[blockIdx.y];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < J.n; i += gridDim.x * blockDim.x)
        data1[start[J.row0 + (((uint32_t)J.c0[i] ^ 0x80000000u) - J.min0)] + place[J.e0 + i]] = J.c1[i];
}

// level-0 values and row pointers (within the relation's own entries), and the
// longest row of every relation
__global__ __launch_bounds__(256) void tries_level0_kernel(const __grid_constant__ TrieJobs A,
                                                           const uint32_t *__restrict__ start,
                                                           int32_t *__restrict__ data0,
                                                           unsigned int *__restrict__ longest) {
    const TrieJob &J = A.j[blockIdx.y];
    uint32_t m = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= J.nrows; v += gridDim.x * blockDim.x) {
        const uint32_t s = start[J.row0 + v];
        J.rowptr[v] = s - J.e0;
        if (v < J.nrows) {
            data0[J.row0 + v] = (int32_t)((J.min0 + v) ^ 0x80000000u);
            m = max(m, start[J.row0 + v + 1] - s);
        }
    }
    m = __reduce_max_sync(AMJ_FULL_MASK, m);
    __shared__ uint32_t wm[8];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) m = max(m, wm[w]);
        if (m > ld_volatile_u32(longest + blockIdx.y)) atomicMax(longest + blockIdx.y, m);
    }
}

// the row pointers of a relation whose repeated rows were dropped
__global__ void tries_rowptr_kernel(const uint32_t *__restrict__ ustart, uint64_t nrows, uint64_t len1,
                                    uint64_t *__restrict__ rowptr) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v <= nrows; v += (uint64_t)gridDim.x * blockDim.x)
        rowptr[v] = v < nrows ? ustart[v] : len1;
}

// The tries of the relations whose rows can be bucketed by counting; *alone gets a
// bit for every other one.  mm[t]: least and greatest values of its columns,
// sign flipped, as build_trie2 takes them (of relations with rows).
static int build_tries2_joint(amj_ctx *ctx, const TrieCols *cols, int count, Trie2 *out, DBuf<char> *block,
                              uint32_t (*mm)[4], bool *mm_read, uint32_t *alone) {
    *alone = (1u << count) - 1;
    TrieJobs A{};
    struct Ctr {
        uint32_t mm[4 * TRIE_JOBS_MAX];
        unsigned int longest[TRIE_JOBS_MAX], nlong;
        unsigned long long distinct[TRIE_JOBS_MAX];
    } h;
    uint64_t nmax = 0, n = 0;
    for (int t = 0; t < count; t++) {
        if (cols[t].n >= (1ull << 31)) return AMJ_OK;
        A.j[t].c0 = cols[t].c0;
        A.j[t].c1 = cols[t].c1;
        A.j[t].n = (uint32_t)cols[t].n;
        nmax = std::max(nmax, cols[t].n);
    }
    if (!nmax) return AMJ_OK;
    DBuf<Ctr> ctr;
    AMJ_TRY(ctr.alloc(ctx, 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(ctr.p, 0, sizeof(Ctr), ctx->stream));
    note_launch(ctx);
    tries_minmax_kernel<<<dim3((unsigned)std::min<uint64_t>((nmax + 255) / 256, (uint64_t)ctx->num_sms * 2), count), 256, 0,
                          ctx->stream>>>(A, ctr.p->mm);
    AMJ_CUDA_TRY(cudaGetLastError());
    AMJ_TRY(read_back(ctx, &h, ctr.p, sizeof(h)));
    // the relations built together: job j of A is relation rel[j]
    int rel[TRIE_JOBS_MAX], jobs = 0;
    uint64_t rows = 0;
    nmax = 0;
    for (int t = 0; t < count; t++) {
        if (!cols[t].n) continue;
        for (int k = 0; k < 4; k++) mm[t][k] = k & 1 ? h.mm[4 * t + k] : ~h.mm[4 * t + k];
        const uint64_t range = (uint64_t)(mm[t][1] - mm[t][0]) + 1;
        if (range > 4 * cols[t].n + 4096 || rows + range >= (1ull << 31) || n + cols[t].n >= (1ull << 31)) continue;
        TrieJob &J = A.j[jobs];
        J.c0 = cols[t].c0;
        J.c1 = cols[t].c1;
        J.n = (uint32_t)cols[t].n;
        J.min0 = mm[t][0];
        J.nrows = (uint32_t)range;
        J.row0 = (uint32_t)rows;
        J.e0 = (uint32_t)n;
        rows += range;
        n += cols[t].n;
        nmax = std::max(nmax, cols[t].n);
        rel[jobs++] = t;
    }
    *mm_read = true;
    if (!jobs) return AMJ_OK;
    // the tries' arrays in one block, the scratch in another
    auto round = [](uint64_t b) { return (b + 255) / 256 * 256; };
    const uint64_t b_data1 = round((n + TRIE_LEVEL1_PAD) * 4), b_src1 = round(n * 4), b_data0 = round(rows * 4);
    uint64_t b_rp = 0;
    for (int j = 0; j < jobs; j++) b_rp += round(((uint64_t)A.j[j].nrows + 1) * 8);
    AMJ_TRY(block->alloc(ctx, b_data1 + b_src1 + b_data0 + b_rp));
    char *at = block->p;
    int32_t *data1 = reinterpret_cast<int32_t *>(at), *src1 = reinterpret_cast<int32_t *>(at + b_data1);
    int32_t *data0 = reinterpret_cast<int32_t *>(at + b_data1 + b_src1);
    at += b_data1 + b_src1 + b_data0;
    RowParts parts;
    for (int j = 0; j < jobs; j++) {
        parts.row[j] = A.j[j].row0;
        A.j[j].rowptr = reinterpret_cast<uint64_t *>(at);
        at += round(((uint64_t)A.j[j].nrows + 1) * 8);
    }
    DBuf<uint32_t> start, place, uniq, longs;
    AMJ_TRY(start.alloc(ctx, rows + 1));
    AMJ_TRY(place.alloc(ctx, n));
    AMJ_TRY(uniq.alloc(ctx, rows));
    AMJ_TRY(longs.alloc(ctx, n / (RK_WARP_MAX + 1) + 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(start.p, 0, (rows + 1) * sizeof(uint32_t), ctx->stream));
    const dim3 grid((unsigned)std::min<uint64_t>((nmax + 255) / 256, (uint64_t)ctx->num_sms * 8), jobs);
    note_launch(ctx);
    tries_count_kernel<<<dim3((unsigned)((nmax + 256 * TRIES_PER_THREAD - 1) / (256 * TRIES_PER_THREAD)), jobs), 256, 0,
                         ctx->stream>>>(A, start.p, place.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    AMJ_TRY(scan_exclusive_u32(ctx, start.p, start.p, rows + 1, nullptr));
    note_launch(ctx);
    tries_scatter_kernel<<<grid, 256, 0, ctx->stream>>>(A, start.p, place.p, data1);
    note_launch(ctx);
    tries_level0_kernel<<<grid, 256, 0, ctx->stream>>>(A, start.p, data0, ctr.p->longest);
    AMJ_CUDA_TRY(cudaGetLastError());
    const unsigned gs = (unsigned)std::min<uint64_t>((rows + RK_SORT_WARPS - 1) / RK_SORT_WARPS,
                                                     (uint64_t)ctx->num_sms * 8);
    note_launch(ctx);
    rk_sort_rows_kernel<<<gs, RK_SORT_WARPS * 32, 0, ctx->stream>>>(start.p, data0, rows, data1, src1, uniq.p, longs.p,
                                                                    &ctr.p->nlong, parts, ctr.p->distinct);
    AMJ_CUDA_TRY(cudaGetLastError());
    if (nmax > RK_WARP_MAX)
        AMJ_TRY(launch_sort_long(ctx, start.p, data0, data1, src1, uniq.p, longs.p, &ctr.p->nlong, parts,
                                 ctr.p->distinct));
    AMJ_TRY(read_back(ctx, &h, ctr.p, sizeof(h)));
    for (int j = 0; j < jobs; j++) {
        Trie2 &o = out[rel[j]];
        const TrieJob &J = A.j[j];
        if (h.longest[j] > RK_BLOCK_MAX) continue;   // unsorted rows
        const uint64_t len1 = h.distinct[j];
        if (len1 == J.n) {
            // views of the block: no context, so they free nothing
            o.data1.p = data1 + J.e0;
            o.data1.n = J.n;
            o.src1.p = src1 + J.e0;
            o.src1.n = J.n;
        } else {
            // repeated rows: the distinct values of every row, moved together
            uint32_t *ustart = uniq.p + J.row0;
            AMJ_TRY(o.data1.alloc(ctx, len1 + TRIE_LEVEL1_PAD));
            AMJ_TRY(o.src1.alloc(ctx, len1));
            AMJ_TRY(scan_exclusive_u32(ctx, ustart, ustart, J.nrows, nullptr));
            note_launch(ctx);
            rk_compact_kernel<<<grid_for(ctx, (uint64_t)J.nrows * 32), 256, 0, ctx->stream>>>(
                start.p + J.row0, ustart, data0 + J.row0, J.nrows, data1, o.data1.p, o.src1.p);
            note_launch(ctx);
            tries_rowptr_kernel<<<grid_for(ctx, (uint64_t)J.nrows + 1), 256, 0, ctx->stream>>>(ustart, J.nrows, len1,
                                                                                             J.rowptr);
            AMJ_CUDA_TRY(cudaGetLastError());
        }
        o.len0 = J.nrows;
        o.len1 = len1;
        o.data0.p = data0 + J.row0;
        o.data0.n = J.nrows;
        o.off0.p = o.rowptr.p = J.rowptr;
        o.off0.n = o.rowptr.n = (uint64_t)J.nrows + 1;
        o.rp_min = (int32_t)(J.min0 ^ 0x80000000u);
        o.rp_count = J.nrows;
        o.range1 = (uint64_t)(mm[rel[j]][3] - mm[rel[j]][2]) + 1;
        *alone &= ~(1u << rel[j]);
    }
    return AMJ_OK;
}

int build_tries2(amj_ctx *ctx, const TrieCols *cols, int count, Trie2 *out, DBuf<char> *block) {
    if (count < 1 || count > TRIE_JOBS_MAX) return fail(AMJ_EINVAL, "tries: bad count");
    uint32_t mm[TRIE_JOBS_MAX][4], alone = 0;
    bool mm_read = false;
    auto build_alone = [&](uint32_t which) {
        for (int t = 0; t < count; t++)
            if ((which >> t) & 1u)
                AMJ_TRY(build_trie2(ctx, cols[t].c0, cols[t].c1, cols[t].n, &out[t], true, -1,
                                    mm_read && cols[t].n ? mm[t] : nullptr));
        return (int)AMJ_OK;
    };
    int rc = build_tries2_joint(ctx, cols, count, out, block, mm, &mm_read, &alone);
    if (rc == AMJ_OK) rc = build_alone(alone);
    if (rc == AMJ_ENOMEM) {
        // one by one, beside nothing else
        for (int t = 0; t < count; t++) out[t] = Trie2();
        block->release();
        rc = build_alone((1u << count) - 1);
    }
    return rc;
}

// ---- N-level tries ----
// Rows are ordered by a stable LSD radix sort of the row permutation, one
// column at a time from the last: items (column value - min) << 32 | row,
// sorted on the value bits only.  Then per level a head flag marks the rows
// whose (l+1)-prefix differs from the previous row's, a scan numbers the
// heads, and a scatter writes the level's values and child offsets.

__global__ void minmax_col_kernel(const int32_t *__restrict__ c, uint64_t n, uint32_t *mm) {
    uint32_t mn = 0xffffffffu, mx = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = (uint32_t)c[i] ^ 0x80000000u;
        mn = min(mn, a);
        mx = max(mx, a);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        mn = min(mn, __shfl_xor_sync(AMJ_FULL_MASK, mn, d));
        mx = max(mx, __shfl_xor_sync(AMJ_FULL_MASK, mx, d));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&mm[0], mn);
        atomicMax(&mm[1], mx);
    }
}

__global__ void pack_col_kernel(const int32_t *__restrict__ c, const uint32_t *__restrict__ perm, uint64_t n,
                                uint32_t mn, uint64_t *__restrict__ items) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = perm ? perm[i] : (uint32_t)i;
        items[i] = ((uint64_t)(((uint32_t)c[r] ^ 0x80000000u) - mn) << 32) | r;
    }
}

__global__ void perm_from_items_kernel(const uint64_t *__restrict__ items, uint64_t n, uint32_t *__restrict__ perm) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        perm[i] = (uint32_t)items[i];
}

__global__ void gather_perm_kernel(const int32_t *__restrict__ c, const uint32_t *__restrict__ perm, uint64_t n,
                                   int32_t *__restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = c[perm ? perm[i] : i];
}

// head[i] = 1 when row i's (l+1)-prefix differs from row i-1's
__global__ void prefix_heads_kernel(int32_t *const *__restrict__ S, int l, uint64_t n, uint32_t *__restrict__ head) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        bool h = i == 0;
        for (int c = 0; c <= l && !h; c++) h = S[c][i] != S[c][i - 1];
        head[i] = h ? 1u : 0u;
    }
}

// level l: values and child offsets at the heads' ranks
__global__ void scatter_level_kernel(const int32_t *__restrict__ Sl, const uint32_t *__restrict__ head,
                                     const uint32_t *__restrict__ rank, const uint32_t *__restrict__ next_rank,
                                     uint64_t n, int32_t *__restrict__ data, uint64_t *__restrict__ off) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!head[i]) continue;
        const uint32_t r = rank[i];
        data[r] = Sl[i];
        off[r] = next_rank ? next_rank[i] : i;
    }
}

int build_trieN(amj_ctx *ctx, const int32_t *const *d_cols, int ncols, uint64_t n, TrieN *out) {
    if (ncols < 1 || ncols > TRIE_MAX_LEVELS) return fail(AMJ_EINVAL, "trie_build_n: 1..8 columns");
    if (n >= (1ull << 32)) return fail(AMJ_EUNSUPPORTED, "trie_build_n: 2^32 or more rows");
    out->levels = ncols;
    // sorted columns
    std::vector<DBuf<int32_t>> S(ncols);
    DBuf<uint32_t> perm;
    if (n > 1) {
        DBuf<uint64_t> a, b;
        DBuf<uint32_t> mm;
        AMJ_TRY(a.alloc(ctx, n));
        AMJ_TRY(b.alloc(ctx, n));
        AMJ_TRY(perm.alloc(ctx, n));
        AMJ_TRY(mm.alloc(ctx, 2 * ncols));
        std::vector<uint32_t> init(2 * ncols);
        for (int c = 0; c < ncols; c++) {
            init[2 * c] = 0xffffffffu;
            init[2 * c + 1] = 0;
        }
        AMJ_CUDA_TRY(cudaMemcpyAsync(mm.p, init.data(), 8 * ncols, cudaMemcpyHostToDevice, ctx->stream));
        for (int c = 0; c < ncols; c++) {
            note_launch(ctx);
            minmax_col_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(d_cols[c], n, mm.p + 2 * c);
        }
        AMJ_CUDA_TRY(cudaGetLastError());
        std::vector<uint32_t> h(2 * ncols);
        AMJ_CUDA_TRY(cudaMemcpyAsync(h.data(), mm.p, 8 * ncols, cudaMemcpyDeviceToHost, ctx->stream));
        AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        bool have_perm = false;
        for (int c = ncols - 1; c >= 0; c--) {
            const uint32_t range = h[2 * c + 1] - h[2 * c];
            int bits = 0;
            while (bits < 32 && (uint64_t)range >> bits) bits++;
            if (bits == 0) continue;   // constant column: the order stays
            note_launch(ctx);
            pack_col_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(d_cols[c], have_perm ? perm.p : nullptr, n,
                                                                      h[2 * c], a.p);
            AMJ_CUDA_TRY(cudaGetLastError());
            uint64_t *sorted = nullptr;
            AMJ_TRY(radix_sort_u64(ctx, a.p, b.p, n, SK_IDENT, 32, 32 + bits, &sorted));
            note_launch(ctx);
            perm_from_items_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sorted, n, perm.p);
            AMJ_CUDA_TRY(cudaGetLastError());
            have_perm = true;
        }
        if (!have_perm) perm.release();
    }
    for (int c = 0; c < ncols; c++) {
        AMJ_TRY(S[c].alloc(ctx, n ? n : 1));
        if (n) {
            note_launch(ctx);
            gather_perm_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(d_cols[c], perm.p, n, S[c].p);
        }
    }
    AMJ_CUDA_TRY(cudaGetLastError());
    // heads and ranks of every level but the last
    const int L = ncols - 1;
    std::vector<DBuf<uint32_t>> head(L), rank(L);
    std::vector<uint32_t> cnt(L, 0);
    DBuf<int32_t *> sp;
    AMJ_TRY(sp.alloc(ctx, ncols));
    std::vector<int32_t *> hp(ncols);
    for (int c = 0; c < ncols; c++) hp[c] = S[c].p;
    AMJ_CUDA_TRY(cudaMemcpyAsync(sp.p, hp.data(), ncols * sizeof(int32_t *), cudaMemcpyHostToDevice, ctx->stream));
    DBuf<uint32_t> totals;
    AMJ_TRY(totals.alloc(ctx, L ? L : 1));
    for (int l = 0; l < L; l++) {
        AMJ_TRY(head[l].alloc(ctx, n ? n : 1));
        AMJ_TRY(rank[l].alloc(ctx, n ? n : 1));
        if (n) {
            note_launch(ctx);
            prefix_heads_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(sp.p, l, n, head[l].p);
            AMJ_CUDA_TRY(cudaGetLastError());
            AMJ_TRY(scan_exclusive_u32(ctx, head[l].p, rank[l].p, n, totals.p + l));
        } else {
            AMJ_CUDA_TRY(cudaMemsetAsync(totals.p + l, 0, 4, ctx->stream));
        }
    }
    if (L) {
        AMJ_CUDA_TRY(cudaMemcpyAsync(cnt.data(), totals.p, 4 * L, cudaMemcpyDeviceToHost, ctx->stream));
        AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    }
    for (int l = 0; l < L; l++) {
        out->len[l] = cnt[l];
        AMJ_TRY(out->data[l].alloc(ctx, cnt[l] ? cnt[l] : 1));
        AMJ_TRY(out->off[l].alloc(ctx, (uint64_t)cnt[l] + 1));
        if (n) {
            note_launch(ctx);
            scatter_level_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(
                S[l].p, head[l].p, rank[l].p, l + 1 < L ? rank[l + 1].p : nullptr, n, out->data[l].p, out->off[l].p);
            AMJ_CUDA_TRY(cudaGetLastError());
        }
        const uint64_t end = l + 1 < L ? (uint64_t)cnt[l + 1] : n;
        AMJ_CUDA_TRY(cudaMemcpyAsync(out->off[l].p + cnt[l], &end, 8, cudaMemcpyHostToDevice, ctx->stream));
        AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    }
    out->len[L] = n;
    out->data[L] = std::move(S[L]);
    return AMJ_OK;
}

}  // namespace amj

using namespace amj;

extern "C" int amj_trie_download_level(const amj_trie *t, int level, int32_t *data, uint64_t *offsets);
extern "C" int amj_trie_save_n(const amj_trie *t, const char *path, const uint32_t *attrs);

extern "C" int amj_trie_build(amj_ctx *ctx, const int32_t *d_c0, const int32_t *d_c1, uint64_t n, amj_trie **out) {
    if (!ctx || !out || (n && (!d_c0 || !d_c1))) return fail(AMJ_EINVAL, "trie_build: null argument");
    *out = nullptr;
    auto *t = new amj_trie();
    t->ctx = ctx;
    int rc = build_trie2(ctx, d_c0, d_c1, n, &t->t);
    if (rc == AMJ_OK) {
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = cuda_fail(e, "trie_build");
    }
    if (rc != AMJ_OK) {
        delete t;
        return rc;
    }
    *out = t;
    return AMJ_OK;
}

extern "C" int amj_trie_view(const amj_trie *t, uint64_t *len0, uint64_t *len1, const int32_t **d_data0,
                             const uint64_t **d_offsets0, const int32_t **d_data1) {
    if (!t) return fail(AMJ_EINVAL, "trie_view: null trie");
    if (t->levels() != 2) return fail(AMJ_EINVAL, "trie_view: not a 2-level trie");
    if (len0) *len0 = t->len(0);
    if (len1) *len1 = t->len(1);
    if (d_data0) *d_data0 = t->data(0);
    if (d_offsets0) *d_offsets0 = t->off(0);
    if (d_data1) *d_data1 = t->data(1);
    return AMJ_OK;
}

extern "C" int amj_trie_download(const amj_trie *t, int32_t *data0, uint64_t *offsets0, int32_t *data1) {
    if (!t || !data0 || !offsets0 || !data1) return fail(AMJ_EINVAL, "trie_download: null argument");
    if (t->levels() != 2) return fail(AMJ_EINVAL, "trie_download: not a 2-level trie");
    AMJ_TRY(amj_trie_download_level(t, 0, data0, offsets0));
    return amj_trie_download_level(t, 1, data1, nullptr);
}

extern "C" void amj_trie_release(amj_trie *t) {
    if (!t) return;
    if (t->ctx) (void)cudaSetDevice(t->ctx->device);
    delete t;
}

// .tr layout (LFTJ-GPU/IndexedTrie.cuh:122-156): uint32 num_attrs, uint64
// data_len[num_attrs], uint32 attr_list[num_attrs], the int32 data of each
// level, then the uint64 offsets of every level but the last
// (data_len[l]+1 entries each).
extern "C" int amj_trie_save(const amj_trie *t, const char *path, uint32_t a0, uint32_t a1) {
    if (!t || !path) return fail(AMJ_EINVAL, "trie_save: null argument");
    if (t->levels() != 2) return fail(AMJ_EINVAL, "trie_save: not a 2-level trie");
    const uint32_t attrs[2] = {a0, a1};
    return amj_trie_save_n(t, path, attrs);
}

extern "C" int amj_trie_load(amj_ctx *ctx, const char *path, amj_trie **out, uint32_t *a0, uint32_t *a1) {
    if (!ctx || !path || !out) return fail(AMJ_EINVAL, "trie_load: null argument");
    *out = nullptr;
    FILE *f = std::fopen(path, "rb");
    if (!f) return fail(AMJ_EIO, std::string("trie_load: cannot open ") + path);
    uint32_t na = 0;
    uint64_t lens[2] = {0, 0};
    uint32_t attrs[2] = {0, 0};
    if (std::fread(&na, 4, 1, f) != 1 || na != 2 || std::fread(lens, 8, 2, f) != 2 || std::fread(attrs, 4, 2, f) != 2) {
        std::fclose(f);
        return fail(AMJ_EIO, "trie_load: bad header (only 2-level tries are supported)");
    }
    const uint64_t l0 = lens[0], l1 = lens[1];
    std::vector<int32_t> d0(l0), d1(l1);
    std::vector<uint64_t> o0(l0 + 1);
    bool ok = (l0 == 0 || std::fread(d0.data(), 4, l0, f) == l0) && (l1 == 0 || std::fread(d1.data(), 4, l1, f) == l1) &&
              std::fread(o0.data(), 8, l0 + 1, f) == l0 + 1;
    std::fclose(f);
    if (!ok || o0[l0] != l1) return fail(AMJ_EIO, "trie_load: truncated or inconsistent file");
    auto *t = new amj_trie();
    t->ctx = ctx;
    t->t.len0 = l0;
    t->t.len1 = l1;
    int rc = t->t.data0.alloc(ctx, l0 ? l0 : 1);
    if (rc == AMJ_OK) rc = t->t.data1.alloc(ctx, l1 ? l1 : 1);
    if (rc == AMJ_OK) rc = t->t.off0.alloc(ctx, l0 + 1);
    if (rc == AMJ_OK && l0 && cudaMemcpyAsync(t->t.data0.p, d0.data(), l0 * 4, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess) rc = AMJ_ECUDA;
    if (rc == AMJ_OK && l1 && cudaMemcpyAsync(t->t.data1.p, d1.data(), l1 * 4, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess) rc = AMJ_ECUDA;
    if (rc == AMJ_OK && cudaMemcpyAsync(t->t.off0.p, o0.data(), (l0 + 1) * 8, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess) rc = AMJ_ECUDA;
    if (rc == AMJ_OK && cudaStreamSynchronize(ctx->stream) != cudaSuccess) rc = AMJ_ECUDA;
    if (rc != AMJ_OK) {
        (void)cudaGetLastError();
        delete t;
        return rc == AMJ_ECUDA ? fail(rc, "trie_load: device copy failed") : rc;
    }
    if (a0) *a0 = attrs[0];
    if (a1) *a1 = attrs[1];
    *out = t;
    return AMJ_OK;
}

extern "C" int amj_trie_build_n(amj_ctx *ctx, const int32_t *const *d_cols, int ncols, uint64_t n, amj_trie **out) {
    if (!ctx || !out || !d_cols) return fail(AMJ_EINVAL, "trie_build_n: null argument");
    if (ncols < 1 || ncols > TRIE_MAX_LEVELS) return fail(AMJ_EINVAL, "trie_build_n: 1..8 columns");
    for (int c = 0; c < ncols && n; c++)
        if (!d_cols[c]) return fail(AMJ_EINVAL, "trie_build_n: null column");
    *out = nullptr;
    auto *t = new amj_trie();
    t->ctx = ctx;
    int rc = build_trieN(ctx, d_cols, ncols, n, &t->tn);
    if (rc == AMJ_OK) {
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = cuda_fail(e, "trie_build_n");
    }
    if (rc != AMJ_OK) {
        delete t;
        return rc;
    }
    *out = t;
    return AMJ_OK;
}

extern "C" int amj_trie_info(const amj_trie *t, int *levels, uint64_t *lens) {
    if (!t) return fail(AMJ_EINVAL, "trie_info: null trie");
    if (levels) *levels = t->levels();
    if (lens)
        for (int l = 0; l < t->levels(); l++) lens[l] = t->len(l);
    return AMJ_OK;
}

extern "C" int amj_trie_download_level(const amj_trie *t, int level, int32_t *data, uint64_t *offsets) {
    if (!t || !data) return fail(AMJ_EINVAL, "trie_download_level: null argument");
    if (level < 0 || level >= t->levels()) return fail(AMJ_EINVAL, "trie_download_level: no such level");
    amj_ctx *ctx = t->ctx;
    const uint64_t n = t->len(level);
    if (n) AMJ_CUDA_TRY(cudaMemcpyAsync(data, t->data(level), n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (offsets && level + 1 < t->levels())
        AMJ_CUDA_TRY(cudaMemcpyAsync(offsets, t->off(level), (n + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream));
    AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return AMJ_OK;
}

// .tr with any number of levels (same layout as amj_trie_save)
extern "C" int amj_trie_save_n(const amj_trie *t, const char *path, const uint32_t *attrs) {
    if (!t || !path || !attrs) return fail(AMJ_EINVAL, "trie_save_n: null argument");
    const int L = t->levels();
    std::vector<std::vector<int32_t>> d(L);
    std::vector<std::vector<uint64_t>> o(L > 1 ? L - 1 : 0);
    for (int l = 0; l < L; l++) {
        d[l].resize(t->len(l));
        if (l + 1 < L) o[l].resize(t->len(l) + 1);
        AMJ_TRY(amj_trie_download_level(t, l, d[l].data(), l + 1 < L ? o[l].data() : nullptr));
    }
    FILE *f = std::fopen(path, "wb");
    if (!f) return fail(AMJ_EIO, std::string("trie_save_n: cannot open ") + path);
    const uint32_t na = (uint32_t)L;
    bool ok = std::fwrite(&na, 4, 1, f) == 1;
    for (int l = 0; l < L && ok; l++) {
        const uint64_t len = t->len(l);
        ok = std::fwrite(&len, 8, 1, f) == 1;
    }
    ok = ok && std::fwrite(attrs, 4, L, f) == (size_t)L;
    for (int l = 0; l < L && ok; l++) ok = d[l].empty() || std::fwrite(d[l].data(), 4, d[l].size(), f) == d[l].size();
    for (int l = 0; l + 1 < L && ok; l++) ok = std::fwrite(o[l].data(), 8, o[l].size(), f) == o[l].size();
    if (std::fclose(f) != 0) ok = false;
    return ok ? AMJ_OK : fail(AMJ_EIO, std::string("trie_save_n: write failed for ") + path);
}

extern "C" int amj_trie_load_n(amj_ctx *ctx, const char *path, amj_trie **out, uint32_t *attrs, int *levels) {
    if (!ctx || !path || !out) return fail(AMJ_EINVAL, "trie_load_n: null argument");
    *out = nullptr;
    FILE *f = std::fopen(path, "rb");
    if (!f) return fail(AMJ_EIO, std::string("trie_load_n: cannot open ") + path);
    uint32_t na = 0;
    uint64_t lens[TRIE_MAX_LEVELS] = {};
    uint32_t at[TRIE_MAX_LEVELS] = {};
    bool ok = std::fread(&na, 4, 1, f) == 1 && na >= 1 && na <= (uint32_t)TRIE_MAX_LEVELS &&
              std::fread(lens, 8, na, f) == na && std::fread(at, 4, na, f) == na;
    std::vector<std::vector<int32_t>> d(ok ? na : 0);
    std::vector<std::vector<uint64_t>> o(ok && na > 1 ? na - 1 : 0);
    for (uint32_t l = 0; ok && l < na; l++) {
        d[l].resize(lens[l]);
        ok = lens[l] == 0 || std::fread(d[l].data(), 4, lens[l], f) == lens[l];
    }
    for (uint32_t l = 0; ok && l + 1 < na; l++) {
        o[l].resize(lens[l] + 1);
        ok = std::fread(o[l].data(), 8, lens[l] + 1, f) == lens[l] + 1 && o[l][lens[l]] == lens[l + 1];
    }
    std::fclose(f);
    if (!ok) return fail(AMJ_EIO, "trie_load_n: bad, truncated or inconsistent file");
    auto *t = new amj_trie();
    t->ctx = ctx;
    t->tn.levels = (int)na;
    int rc = AMJ_OK;
    for (uint32_t l = 0; rc == AMJ_OK && l < na; l++) {
        t->tn.len[l] = lens[l];
        rc = t->tn.data[l].alloc(ctx, lens[l] ? lens[l] : 1);
        if (rc == AMJ_OK && lens[l] &&
            cudaMemcpyAsync(t->tn.data[l].p, d[l].data(), lens[l] * 4, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess)
            rc = AMJ_ECUDA;
        if (rc == AMJ_OK && l + 1 < na) {
            rc = t->tn.off[l].alloc(ctx, lens[l] + 1);
            if (rc == AMJ_OK && cudaMemcpyAsync(t->tn.off[l].p, o[l].data(), (lens[l] + 1) * 8, cudaMemcpyHostToDevice,
                                                ctx->stream) != cudaSuccess)
                rc = AMJ_ECUDA;
        }
    }
    if (rc == AMJ_OK && cudaStreamSynchronize(ctx->stream) != cudaSuccess) rc = AMJ_ECUDA;
    if (rc != AMJ_OK) {
        (void)cudaGetLastError();
        delete t;
        return rc == AMJ_ECUDA ? fail(rc, "trie_load_n: device copy failed") : rc;
    }
    if (attrs)
        for (uint32_t l = 0; l < na; l++) attrs[l] = at[l];
    if (levels) *levels = (int)na;
    *out = t;
    return AMJ_OK;
}
