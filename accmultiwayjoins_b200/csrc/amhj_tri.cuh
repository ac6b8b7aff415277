// Triangle queries of a batch, joined flat.
//
// The TRI plan over one edge relation R is R(a,b), then R(b,c) looked up by b,
// then the pair-key filter R(a,c).  Both later levels read the same relation,
// so the candidates c may as well come from a's rows with (b,c) as the filter:
// the same rows of the same two indexes, multiplicities included.  Each probe
// row takes the shorter of its two candidate lists.  On a graph given with
// its hubs first (R-MAT, edges from the lower to the higher id) most of the
// wedges hang on one hub, and the shorter lists leave half of the candidates
// (0.70 G of 1.35 G).  (The single-query operator joins a degree-ranked copy instead;
// a batch joins its relations as given, since a replayed batch reads them
// again.)
// A unit is TRI_CHUNK candidates.  A warp loads the rows of its unit 32 at a
// time, one a lane, and hands out their candidates one a lane: the lane whose
// row starts at a candidate marks it in a 32-bit word, so the owner of a
// candidate is a population count and not a search.  The filter is one 32-byte
// bucket head (two bounds and three rows) instead of two bounds and then the
// rows' columns.  There is no frontier, no task and no wait: every candidate
// is one filter lookup.  Bound by the random sectors of the heads.
// Measured, 54 triangle queries of 10K to 1M edges, 107 M triangles: the probe
// takes 7.3 ms; through the frontier DFS, with b's list alone and the pair
// filter's bounds and columns read one by one, it took 40.2 ms.
#pragma once
#include "amhj_kernel.cuh"

namespace amj {

constexpr uint32_t TRI_CHUNK = 1024;
constexpr int TRI_THREADS = 256;
constexpr int TRI_WARPS = TRI_THREADS / 32;

// The shorter candidate list of probe row i: its start and length in the
// index of lv[0], keyed by a or (a = false) by b.
__device__ __forceinline__ uint32_t tri_side(const ProbePlan &P, int32_t a, int32_t b, uint32_t &s, bool &by_a) {
    const LevelDesc &lv = P.lv[0];
    const uint32_t ha = (uint32_t)a & lv.mask, hb = (uint32_t)b & lv.mask;
    const uint32_t sa = lv.buc_ptrs[ha], na = lv.buc_ptrs[ha + 1] - sa;
    const uint32_t sb = lv.buc_ptrs[hb], nb = lv.buc_ptrs[hb + 1] - sb;
    by_a = na < nb;
    s = by_a ? sa : sb;
    return by_a ? na : nb;
}

// column of attribute 0 (a) or 1 (b) of the probe relation
__device__ __forceinline__ const int32_t *tri_col(const ProbePlan &P, int attr) {
    return P.probe_col[P.probe_attr[0] == attr ? 0 : 1];
}

struct TriLaunch {
    const ProbePlan *plans;
    const unsigned long long *tri_base;   // first triangle unit of every query (nq + 1 entries)
    unsigned long long *next;             // unit counter
    unsigned long long *q_count;
    unsigned long long *q_checksum;
    uint32_t nq;
};

struct TriWarp {
    unsigned long long hab[32];   // hash prefix of (a, b)
    int4 ent[32];                 // list start minus the candidates before it, key, other vertex
};

__global__ __launch_bounds__(TRI_THREADS) void batch_tri_kernel(const TriLaunch T) {
    __shared__ TriWarp smem[TRI_WARPS];
    const int lane = threadIdx.x & 31;
    TriWarp &W = smem[threadIdx.x >> 5];
    const unsigned lt = lanemask_lt(), le = lt | (1u << lane);
    const unsigned long long total = T.tri_base[T.nq];
    unsigned long long cnt = 0, chk = 0;
    int cur = -1;
    auto flush = [&]() {
        const unsigned long long c = warp_sum(cnt), h = warp_sum(chk);
        if (lane == 0 && cur >= 0 && c) {
            atomicAdd(&T.q_count[cur], c);
            atomicAdd(&T.q_checksum[cur], h);
        }
        cnt = chk = 0;
    };
    while (true) {
        unsigned long long u = 0;
        if (lane == 0) u = atomicAdd(T.next, 1ull);
        u = __shfl_sync(AMJ_FULL_MASK, u, 0);
        if (u >= total) break;
        const int q = (int)warp_row_of(T.tri_base, T.nq, u, lane);
        if (q != cur) {
            flush();
            cur = q;
        }
        const ProbePlan &P = T.plans[q];
        const unsigned long long *E = P.l0_start;
        const uint64_t rows = P.row_hi;
        const unsigned long long g0 = E[0] + (u - T.tri_base[q]) * TRI_CHUNK, end = E[rows];
        const unsigned long long g1 = g0 + TRI_CHUNK < end ? g0 + TRI_CHUNK : end;
        const uint64_t rlo = warp_row_of(E, rows, g0, lane), rhi = warp_row_of(E, rows, g1 - 1, lane) + 1;
        const int32_t *ca = tri_col(P, 0), *cb = tri_col(P, 1);
        const int32_t *key0 = P.lv[0].col[0], *val0 = P.lv[0].col[1];
        const LevelDesc &fl = P.lv[1];
        const BucketHead *heads = P.tri_heads;
        for (uint64_t r0 = rlo; r0 < rhi; r0 += 32) {
            const uint64_t r = r0 + lane;
            uint32_t sz = 0, s = 0;
            int32_t a = 0, b = 0;
            bool by_a = false;
            if (r < rhi) {
                const unsigned long long e0 = E[r], e1 = E[r + 1];
                const unsigned long long lo = e0 > g0 ? e0 : g0, hi = e1 < g1 ? e1 : g1;
                if (hi > lo) {
                    a = ca[r];
                    b = cb[r];
                    tri_side(P, a, b, s, by_a);
                    s += (uint32_t)(lo - e0);
                    sz = (uint32_t)(hi - lo);
                }
            }
            const uint32_t incl = warp_inclusive_scan(sz, lane), excl = incl - sz;
            const uint32_t tot = __shfl_sync(AMJ_FULL_MASK, incl, 31);
            const unsigned live = __ballot_sync(AMJ_FULL_MASK, sz > 0);
            __syncwarp();
            if (sz) {
                const int at = __popc(live & lt);
                W.ent[at] = make_int4((int)(s - excl), by_a ? a : b, by_a ? b : a, 0);
                W.hab[at] = amj_hash_step(amj_hash_step(AMJ_CHECKSUM_SEED, a), b);
            }
            __syncwarp();
            int before = -1;   // rows started before this step, minus one
            for (uint32_t j0 = 0; j0 < tot; j0 += 32) {
                const unsigned starts =
                    __reduce_or_sync(AMJ_FULL_MASK, sz && excl - j0 < 32u ? 1u << (excl - j0) : 0u);
                const int o = before + __popc(starts & le);
                before += __popc(starts);
                const uint32_t j = j0 + lane;
                if (j >= tot) continue;
                const int4 e = W.ent[o];
                const uint32_t slot = (uint32_t)e.x + j;
                const int32_t c = val0[slot];
                if (key0[slot] != e.y) continue;
                const uint32_t h = hash_pair(e.z, c) & fl.mask;
                uint32_t m = 0, rs, re;
                if (heads) {
                    uint32_t w[8];
                    load_head(heads + h, w);
                    rs = w[0];
                    re = w[1];
                    const uint32_t n = re - rs;
#pragma unroll
                    for (int i = 0; i < HEAD_ROWS; i++)
                        m += ((uint32_t)i < n && (int32_t)w[2 + 2 * i] == e.z && (int32_t)w[3 + 2 * i] == c) ? 1u : 0u;
                    rs += HEAD_ROWS;
                } else {
                    rs = fl.buc_ptrs[h];
                    re = fl.buc_ptrs[h + 1];
                }
                for (; rs < re; rs++) m += (fl.col[0][rs] == e.z && fl.col[1][rs] == c) ? 1u : 0u;
                if (m) {
                    cnt += m;
                    chk += m * amj_hash_step(W.hab[o], c);
                }
            }
        }
    }
    flush();
}

// heads of the pair indexes of the triangle queries
struct TriHeadJob {
    const uint32_t *bp;
    const int32_t *c0, *c1;
    unsigned long long first;   // first head
};

__global__ void batch_tri_heads_kernel(const TriHeadJob *__restrict__ jobs, const unsigned long long *__restrict__ first,
                                       uint32_t njobs, uint64_t total, BucketHead *__restrict__ heads) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = njobs;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (first[mid] <= t) lo = mid;
            else hi = mid;
        }
        const TriHeadJob &J = jobs[lo];
        const uint64_t h = t - J.first;
        BucketHead o;
        o.s = J.bp[h];
        o.e = J.bp[h + 1];
#pragma unroll
        for (int i = 0; i < HEAD_ROWS; i++) {
            const bool in = o.s + i < o.e;
            o.kp[2 * i] = in ? J.c0[o.s + i] : 0;
            o.kp[2 * i + 1] = in ? J.c1[o.s + i] : 0;
        }
        heads[t] = o;
    }
}

}  // namespace amj
