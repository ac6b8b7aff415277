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
// candidate is a population count and not a search.  Most candidates close no
// triangle (107 M of 697 M do), so a word a bucket, with a bit for each row's pair
// hash, turns them down first: 4 bytes a candidate, which the L1 and L2 hold.
// Those that pass wait in a ring until 32 of them look up their bucket's head (two
// bounds and three rows, 32 bytes) together.  There is no frontier, no task and
// no wait on another warp.  Bound by the latency of the dependent loads and by
// instructions (half of the issue slots before the bits).
// Measured, 54 triangle queries of 10K to 1M edges, 107 M triangles: the probe
// takes 5.2 ms; 7.2 with a head lookup a candidate (6.8 to 8.8 with 16-byte heads
// of twice as many buckets); 40.2 through the frontier DFS, with b's list alone and
// the pair filter's bounds and columns read one by one.  Two candidates a
// lane and step: 5.2.
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
    // candidates that passed the filter's bits, a ring of 64
    unsigned long long qhab[64];
    int4 q[64];                   // other vertex, candidate, pair hash
};

// six blocks an SM (four, five, eight: 5.5, 5.4, 5.4 ms)
__global__ __launch_bounds__(TRI_THREADS, 6) void batch_tri_kernel(const TriLaunch T) {
    __shared__ TriWarp smem[TRI_WARPS];
    const int lane = threadIdx.x & 31;
    TriWarp &W = smem[threadIdx.x >> 5];
    const unsigned lt = lanemask_lt(), le = lt | (1u << lane);
    const unsigned long long total = T.tri_base[T.nq];
    unsigned long long cnt = 0, chk = 0;
    int cur = -1;
    uint32_t qh = 0, qn = 0;   // the ring's first entry and their number
    // look up the ring's first n <= 32 entries in the current query's filter
    auto drain = [&](uint32_t n) {
        if ((uint32_t)lane < n) {
            const ProbePlan &P = T.plans[cur];
            const LevelDesc &fl = P.lv[1];
            const int4 x = W.q[(qh + lane) & 63];
            const uint32_t h = (uint32_t)x.z & fl.mask;
            uint32_t m = 0, rs, re;
            if (P.tri_heads) {
                uint32_t w[8];
                load_head(P.tri_heads + h, w);
                rs = w[0];
                re = w[1];
                const uint32_t k = re - rs;
#pragma unroll
                for (int i = 0; i < HEAD_ROWS; i++)
                    m += ((uint32_t)i < k && (int32_t)w[2 + 2 * i] == x.x && (int32_t)w[3 + 2 * i] == x.y) ? 1u : 0u;
                rs = k > (uint32_t)HEAD_ROWS ? rs + HEAD_ROWS : re;
            } else {
                rs = fl.buc_ptrs[h];
                re = fl.buc_ptrs[h + 1];
            }
            for (; rs < re; rs++) m += (fl.col[0][rs] == x.x && fl.col[1][rs] == x.y) ? 1u : 0u;
            if (m) {
                cnt += m;
                chk += m * amj_hash_step(W.qhab[(qh + lane) & 63], x.y);
            }
        }
        __syncwarp();
        qh += n;
        qn -= n;
    };
    auto flush = [&]() {
        if (qn) drain(qn);
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
        const uint32_t *bits = P.tri_bits;
        const uint32_t mask1 = P.lv[1].mask;
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
                bool hit = false;
                int4 e = make_int4(0, 0, 0, 0);
                int32_t c = 0;
                uint32_t h = 0;
                if (j < tot) {
                    e = W.ent[o];
                    const uint32_t slot = (uint32_t)e.x + j;
                    c = val0[slot];
                    h = hash_pair(e.z, c);
                    hit = key0[slot] == e.y && (!bits || ((__ldg(bits + (h & mask1)) >> (h >> 27)) & 1u));
                }
                const unsigned hits = __ballot_sync(AMJ_FULL_MASK, hit);
                if (hit) {
                    const uint32_t at = (qh + qn + __popc(hits & lt)) & 63;
                    W.q[at] = make_int4(e.z, c, (int)h, 0);
                    W.qhab[at] = W.hab[o];
                }
                __syncwarp();
                qn += __popc(hits);
                if (qn >= 32) drain(32);
            }
        }
    }
    flush();
}

// Rows of a bucket that its filter word is made of; longer buckets get a word of
// ones.  One thread reads them one by one: an edge repeated a million times
// kept it (and the batch) busy for 89 ms.
constexpr uint32_t TRI_BITS_ROWS = 64;

// heads of the pair indexes of the triangle queries
struct TriHeadJob {
    const uint32_t *bp;
    const int32_t *c0, *c1;
    unsigned long long first;   // first head
};

__global__ void batch_tri_heads_kernel(const TriHeadJob *__restrict__ jobs, const unsigned long long *__restrict__ first,
                                       uint32_t njobs, uint64_t total, BucketHead *__restrict__ heads,
                                       uint32_t *__restrict__ bits) {
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
        // a long bucket's word would have nearly every bit set, or its rows are
        // copies of one pair, which never set them all: it turns nothing down
        uint32_t w = o.e - o.s > TRI_BITS_ROWS ? ~0u : 0u;
        for (uint32_t i = o.s; i < o.e && w != ~0u; i++) w |= 1u << (hash_pair(J.c0[i], J.c1[i]) >> 27);
        bits[t] = w;
    }
}

}  // namespace amj
