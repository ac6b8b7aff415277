// ALFTJ 4-clique: the FOUR pattern A(0,1) B(1,2) C(2,3) D(0,3) E(0,2) F(1,3)
// (MHJ-GPU/exec_AMHJ.cu:50-69) as a leapfrog triejoin over one edge
// relation, attribute order a, b, c, d:
//   b in N(a);   c in N(a) ∩ N(b) = C(a,b);   d in C(a,b) ∩ N(c)
// where N(v) is v's child list in the relation's trie.  The reference's LFTJ
// stops at three attributes (LFTJ-GPU/config.h:16-17); this is its 4-attribute
// form for the FOUR query, the answer AMHJ FOUR gives on the same relation.
//
// Persistent warps claim 32 edges (a,b) at a time.
//  * An edge whose shorter list has at most 16 values is joined by its own
//    lane: C(a,b) by a merge into registers, then C(a,b) ∩ N(c) for every c
//    in it (merge, or per-value galloping search when N(c) is much longer).
//  * Longer edges are joined by the whole warp: C(a,b) by the warp
//    intersection, compacted with ballots into the warp's scratch area; then
//    the warp's lanes take 32 values c at a time, each intersecting C(a,b)
//    with N(c) on its own when the shorter side has at most 32 values, the
//    others one after another by the whole warp.
// Lists are strictly increasing (relations without duplicate edges, as for
// the triangle).
#include "lftj_common.cuh"

#include <algorithm>
#include <cstddef>

namespace amj {

struct C4Args {
    const int32_t *src, *dst;   // the trie's level-1 entries: edge (src[j], dst[j])
    uint64_t n;
    TrieRef T;
    unsigned long long *cursor, *count, *checksum, *out_cursor;
    int32_t *out[4];
    uint64_t out_cap;
    int32_t *scratch;           // per warp: scratch_cap values
    uint64_t scratch_cap;
    int sorted_out;             // degree-ordered copy of an oriented relation: list tuples increasing
};

__device__ __forceinline__ uint64_t umin(uint64_t x, uint64_t y) { return x < y ? x : y; }
__device__ __forceinline__ uint64_t umax(uint64_t x, uint64_t y) { return x < y ? y : x; }

constexpr int C4_LANE_MAX = 16;   // shorter list of a lane-joined edge
constexpr int C4_LANE_PAIR = 32;  // shorter list of a lane-joined (C, N(c)) pair

// One 4-clique: count, checksum, and in write mode one output row.
template <bool WRITE>
__device__ __forceinline__ void c4_emit(const C4Args &A, int32_t a, int32_t b, int32_t c, int32_t d, uint64_t habc,
                                        unsigned long long &cnt, unsigned long long &chk) {
    cnt++;
    if (A.sorted_out) {
        // sorting network of four
        int32_t t;
        if (a > b) { t = a; a = b; b = t; }
        if (c > d) { t = c; c = d; d = t; }
        if (a > c) { t = a; a = c; c = t; }
        if (b > d) { t = b; b = d; d = t; }
        if (b > c) { t = b; b = c; c = t; }
        chk += amj_hash_step(amj_hash_step(amj_hash_step(amj_hash_step(AMJ_CHECKSUM_SEED, a), b), c), d);
    } else {
        chk += amj_hash_step(habc, d);
    }
    if (WRITE) {
        const unsigned long long p = atomicAdd(A.out_cursor, 1ull);
        if (p < A.out_cap) {
            A.out[0][p] = a;
            A.out[1][p] = b;
            A.out[2][p] = c;
            A.out[3][p] = d;
        }
    }
}

// Lane-local intersection of strictly increasing X[0,nx) and Y[0,ny): f(v)
// for each common value.  A merge when the lengths are close; otherwise every
// value of the shorter list is looked up in the longer one by galloping from
// the previous position.
template <class XP, class F>
__device__ __forceinline__ void lane_intersect(XP X, uint64_t nx, const int32_t *Y, uint64_t ny, F &&f) {
    if (nx == 0 || ny == 0) return;
    if (ny <= 8 * nx) {
        uint64_t p = 0, q = 0;
        while (p < nx && q < ny) {
            const int32_t x = X[p], y = Y[q];
            if (x == y) {
                f(x);
                p++;
                q++;
            } else if (x < y) {
                p++;
            } else {
                q++;
            }
        }
        return;
    }
    uint64_t q = 0;
    for (uint64_t p = 0; p < nx && q < ny; p++) {
        const int32_t x = X[p];
        // gallop: smallest q' >= q with Y[q'] >= x
        uint64_t step = 1, lo = q, hi = q;
        while (hi < ny && Y[hi] < x) {
            lo = hi + 1;
            hi = q + step;
            step <<= 1;
        }
        if (hi > ny) hi = ny;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (Y[mid] < x) lo = mid + 1;
            else hi = mid;
        }
        q = lo;
        if (q < ny && Y[q] == x) {
            f(x);
            q++;
        }
    }
}

template <bool WRITE>
__global__ __launch_bounds__(256) void lftj_clique4_kernel(const __grid_constant__ C4Args A) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    int32_t *buf = A.scratch + gw * A.scratch_cap;
    const int32_t *D1 = A.T.data1;
    unsigned long long cnt = 0, chk = 0;
    while (true) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(A.cursor, 32ull);
        base = __shfl_sync(AMJ_FULL_MASK, base, 0);
        if (base >= A.n) break;
        const uint64_t j = base + lane;
        const bool valid = j < A.n;
        int32_t a = 0, b = 0;
        uint64_t ta = 0, ea = 0, tb = 0, eb = 0;
        if (valid) {
            a = A.src[j];
            b = A.dst[j];
            child_range(A.T, a, ta, ea);
            if (ea > ta) child_range(A.T, b, tb, eb);
        }
        const uint64_t la = ea - ta, lb = eb - tb;
        const bool active = valid && la && lb;
        const bool small = active && umin(la, lb) <= (uint64_t)C4_LANE_MAX;
        const uint64_t hab = amj_hash_step(amj_hash_step(AMJ_CHECKSUM_SEED, a), b);
        // ---- short edges: one lane each
        if (small) {
            int32_t cl[C4_LANE_MAX];
            int m = 0;
            lane_intersect(D1 + (la <= lb ? ta : tb), umin(la, lb), D1 + (la <= lb ? tb : ta), umax(la, lb),
                           [&](int32_t v) { cl[m++] = v; });
            for (int i = 0; i < m; i++) {
                const int32_t c = cl[i];
                uint64_t tc, ec;
                child_range(A.T, c, tc, ec);
                const uint64_t habc = amj_hash_step(hab, c);
                lane_intersect(cl, (uint64_t)m, D1 + tc, ec - tc,
                               [&](int32_t d) { c4_emit<WRITE>(A, a, b, c, d, habc, cnt, chk); });
            }
        }
        // ---- long edges: the whole warp, one edge after another
        unsigned big = __ballot_sync(AMJ_FULL_MASK, active && !small);
        while (big) {
            const int l = __ffs(big) - 1;
            big &= big - 1;
            const int32_t wa = __shfl_sync(AMJ_FULL_MASK, a, l), wb = __shfl_sync(AMJ_FULL_MASK, b, l);
            const uint64_t wta = __shfl_sync(AMJ_FULL_MASK, ta, l), wea = __shfl_sync(AMJ_FULL_MASK, ea, l);
            const uint64_t wtb = __shfl_sync(AMJ_FULL_MASK, tb, l), web = __shfl_sync(AMJ_FULL_MASK, eb, l);
            const uint64_t whab = __shfl_sync(AMJ_FULL_MASK, hab, l);
            // C(a,b) into the scratch area (at most the shorter list, which fits it)
            uint64_t m = 0;
            warp_intersect_rounds(D1 + wta, wea - wta, D1 + wtb, web - wtb, lane, [&](bool hit, int32_t v) {
                const unsigned hm = __ballot_sync(AMJ_FULL_MASK, hit);
                if (hit) buf[m + __popc(hm & lt)] = v;
                m += __popc(hm);
            });
            __syncwarp();
            for (uint64_t i0 = 0; i0 < m; i0 += 32) {
                const uint64_t i = i0 + lane;
                const bool has = i < m;
                int32_t c = 0;
                uint64_t tc = 0, ec = 0;
                if (has) {
                    c = buf[i];
                    child_range(A.T, c, tc, ec);
                }
                const uint64_t lc = ec - tc;
                const uint64_t habc = amj_hash_step(whab, c);
                const bool pair = has && lc;
                const bool lone = pair && umin(lc, m) <= (uint64_t)C4_LANE_PAIR;
                if (lone) {
                    if (m <= lc) lane_intersect(buf, m, D1 + tc, lc,
                                                [&](int32_t d) { c4_emit<WRITE>(A, wa, wb, c, d, habc, cnt, chk); });
                    else lane_intersect(D1 + tc, lc, buf, m,
                                        [&](int32_t d) { c4_emit<WRITE>(A, wa, wb, c, d, habc, cnt, chk); });
                }
                unsigned wide = __ballot_sync(AMJ_FULL_MASK, pair && !lone);
                while (wide) {
                    const int l2 = __ffs(wide) - 1;
                    wide &= wide - 1;
                    const int32_t wc = __shfl_sync(AMJ_FULL_MASK, c, l2);
                    const uint64_t wtc = __shfl_sync(AMJ_FULL_MASK, tc, l2), wec = __shfl_sync(AMJ_FULL_MASK, ec, l2);
                    const uint64_t whabc = __shfl_sync(AMJ_FULL_MASK, habc, l2);
                    warp_intersect(buf, m, D1 + wtc, wec - wtc, lane,
                                   [&](int32_t d) { c4_emit<WRITE>(A, wa, wb, wc, d, whabc, cnt, chk); });
                }
            }
            __syncwarp();
        }
    }
    cnt = warp_sum(cnt);
    chk = warp_sum(chk);
    if (lane == 0 && cnt) {
        atomicAdd(A.count, cnt);
        atomicAdd(A.checksum, chk);
    }
}


struct C4Counters {
    unsigned long long cursor, count, checksum, out_cursor, max_deg;
};

// One 4-clique pass over the trie T of the edge relation: count and checksum,
// and the tuples when `out` is given (out_cap rows).
// ---- 4-cliques from triangle matrices (degree-ranked copy) ----
// Over the degree-ranked copy every 4-clique has one vertex a of the lowest
// rank, and is a triangle inside N+(a).  The wedge kernel in matrix mode
// records the triangles through a as bits of a's matrix, whose rows and
// columns are a's children by vertex id; c4m_mirror_kernel then makes row x
// hold bit y for every y > x adjacent to x.  The 4-cliques through (a, x) are
// the adjacent pairs y < z among the bits of row x.
// Numbering by id (not by rank) lists x < y < z in the order of the result
// tuple, into which only a has to be put at its place pa: the tuple hash of
// (x, y), with a when it comes before z, is one prefix for all z, so a tuple
// costs one hash step (a before z) or two (a last) and no sorting.
// Persistent warps claim 32 level-1 entries (a, x) at a time.  The bits of
// row x become a list; 32 values y of it (their prefixes in shared memory)
// meet 32 values z at a time: each lane takes one z and collects its adjacency
// to the 32 y as a mask (a word of row y a step, the same for neighbouring
// lanes).  On the skewed R-MAT graphs over half of the pairs are adjacent
// (55 % at scales 18 and 19), so the masks are dense; their bits go to a list
// of at most 1024 pairs, which the lanes hash (and write) 32 at a time.
// Measured, R-MAT scale 20 (12 G 4-cliques): 53 ms; each lane hashing its own
// mask's bits (18 of 32 lanes active) 70 ms; three or five blocks per SM
// instead of four 57 and 58 ms.  The kernel is bound by the integer pipe (two
// 64-bit mixes a tuple) and the issue slots.  R-MAT scale 22 (94 G
// 4-cliques): 337 ms, against 802 ms for the form in rank order, which
// ANDed whole rows, queued their bits, and sorted and hashed every tuple in
// three steps.
constexpr int C4M_THREADS = 256;
constexpr int C4M_WARPS = C4M_THREADS / 32;
constexpr uint32_t C4M_MAX_DEG = 1024;

struct C4MWarp {
    uint64_t p[2][32];                // prefixes of the 32 y in progress, with a and without
    int2 z[32];                       // the 32 z: id, and byte offset in p of its prefixes
    int32_t yid[32];
    uint16_t ylist[C4M_MAX_DEG + 8];  // the bits of row x, then zeros
    uint16_t q[32 * 32 + 32];         // adjacent pairs: slot of y << 3 | lane of z << 11
};
static_assert(sizeof(C4MWarp) % 16 == 0 && offsetof(C4MWarp, ylist) % 16 == 0, "ylist is read 16 bytes at a time");

struct C4MArgs {
    const int32_t *src1;     // rank a of every level-1 entry
    const int32_t *inv;      // rank -> vertex id
    const int32_t *sid;      // every child list of level 1 by vertex id
    const uint16_t *pa;      // place of a's id among its children's
    TrieRef T;
    const uint64_t *moff;    // first matrix word of every rank
    const uint32_t *mtx;
    uint64_t n;
    unsigned long long *cursor, *count, *checksum, *out_cursor;
    int32_t *out[4];
    uint64_t out_cap;
};

template <bool WRITE>
__global__ __launch_bounds__(C4M_THREADS, 4) void lftj_clique4_matrix_kernel(const __grid_constant__ C4MArgs A) {
    __shared__ C4MWarp smem[C4M_WARPS];
    const int lane = threadIdx.x & 31;
    C4MWarp &S = smem[threadIdx.x >> 5];
    unsigned long long cnt = 0, chk = 0;
    while (true) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(A.cursor, 32ull);
        at = __shfl_sync(AMJ_FULL_MASK, at, 0);
        if (at >= A.n) break;
        const uint64_t j = at + lane;
        int32_t a = -1;
        uint32_t deg = 0, row = 0;
        uint64_t ta = 0, mbase = 0;
        if (j < A.n) {
            a = A.src1[j];
            uint64_t te;
            child_range(A.T, a, ta, te);
            deg = (uint32_t)(te - ta);
            row = (uint32_t)(j - ta);
            mbase = A.moff[a];
        }
        // x needs two children after it
        unsigned todo = __ballot_sync(AMJ_FULL_MASK, row + 2 < deg);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t wl = (__shfl_sync(AMJ_FULL_MASK, deg, l) + 31) / 32;
            const uint32_t x = __shfl_sync(AMJ_FULL_MASK, row, l);
            const uint32_t *M = A.mtx + __shfl_sync(AMJ_FULL_MASK, mbase, l);
            // the bits above x of row x, one word per lane
            uint32_t rx = (uint32_t)lane < wl && (uint32_t)lane >= x / 32 ? M[x * wl + lane] : 0u;
            if ((uint32_t)lane == x / 32) rx &= ~1u << (x & 31);
            const uint32_t nyl = __popc(rx);
            const uint32_t yincl = warp_inclusive_scan(nyl, lane);
            const uint32_t ny = __shfl_sync(AMJ_FULL_MASK, yincl, 31);
            if (ny < 2) continue;
            const int32_t al = __shfl_sync(AMJ_FULL_MASK, a, l);
            const int32_t *sid = A.sid + __shfl_sync(AMJ_FULL_MASK, ta, l);
            const int32_t ida = A.inv[al], xid = sid[x];
            const uint32_t pa = A.pa[al];
            __syncwarp();
            {
                uint32_t p = yincl, m = rx;
                while (m) {
                    const uint32_t b = 31 - __clz(m);
                    m ^= 1u << b;
                    S.ylist[--p] = (uint16_t)(lane * 32 + b);
                }
                if (lane < 8) S.ylist[ny + lane] = 0;
            }
            __syncwarp();
            // prefixes of x: e1 with a when it comes before x; e2 always with a
            uint64_t e1 = amj_hash_step(AMJ_CHECKSUM_SEED, x < pa ? xid : ida), e2;
            if (x < pa) e2 = amj_hash_step(e1, ida);
            else e1 = e2 = amj_hash_step(e1, xid);
            for (uint32_t y0 = 0; y0 + 1 < ny; y0 += 32) {
                const uint32_t nb = min(32u, ny - y0);
                if ((uint32_t)lane < nb) {
                    // slot nb - 1 - i holds the prefixes of y i; where a
                    // comes before x both hold a (e1 = e2 and y >= pa)
                    const uint32_t y = S.ylist[y0 + lane];
                    const int32_t yid = sid[y];
                    const uint64_t p2 = amj_hash_step(e1, yid);
                    S.p[1][nb - 1 - lane] = p2;
                    S.p[0][nb - 1 - lane] = amj_hash_step(y < pa ? p2 : e2, y < pa ? ida : yid);
                    if (WRITE) S.yid[nb - 1 - lane] = yid;
                }
                __syncwarp();
                for (uint32_t z0 = y0; z0 < ny; z0 += 32) {
                    const bool valid = z0 + lane < ny;
                    const uint32_t z = valid ? S.ylist[z0 + lane] : 0u;
                    // rows by 32-bit byte offsets from this lane's column of words
                    const char *col = reinterpret_cast<const char *>(M + (z >> 5));
                    const uint32_t sh = 31 - (z & 31);
                    // bit nb - 1 - i of m: z is adjacent to y i
                    uint32_t m = 0;
                    for (uint32_t i = 0; i < nb; i += 8) {
                        const uint4 y8 = *reinterpret_cast<const uint4 *>(S.ylist + y0 + i);
                        const uint32_t yy[4] = {y8.x, y8.y, y8.z, y8.w};
                        uint32_t w[8];
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            w[k] = *reinterpret_cast<const uint32_t *>(
                                col + (size_t)(((yy[k / 2] >> (16 * (k & 1))) & 0xffffu) * (wl * 4)));
#pragma unroll
                        for (int k = 0; k < 8; k++) m = __funnelshift_l(w[k] << sh, m, 1);
                    }
                    m >>= (0u - nb) & 7u;   // the zeros after the list
                    if (z0 == y0) m &= (uint32_t)lane ? ~0u << (nb > (uint32_t)lane ? nb - lane : 0u) : 0u;   // y before z
                    if (!valid) m = 0;
                    const uint32_t nh = __popc(m);
                    const uint32_t incl = warp_inclusive_scan(nh, lane);
                    uint32_t qn = __shfl_sync(AMJ_FULL_MASK, incl, 31);
                    if (!qn) continue;
                    if (lane == 0) cnt += qn;
                    // a comes after z where z < pa: prefixes without a
                    S.z[lane] = make_int2(sid[z], z < pa ? (int)sizeof(S.p[0]) : 0);
                    {
                        uint16_t *qp = S.q + (incl - nh);
                        while (m) {
                            const uint32_t b = 31 - __clz(m);
                            m ^= 1u << b;
                            *qp++ = (uint16_t)((uint32_t)lane << 11 | b << 3);
                        }
                    }
                    unsigned long long pos = 0;
                    if (WRITE) {
                        if (lane == 0) pos = atomicAdd(A.out_cursor, (unsigned long long)qn);
                        pos = __shfl_sync(AMJ_FULL_MASK, pos, 0) + lane;
                    }
                    __syncwarp();
#pragma unroll 2
                    for (uint32_t i = lane; i < qn; i += 32) {
                        const uint32_t e = S.q[i];
                        const int2 zz = *reinterpret_cast<const int2 *>(reinterpret_cast<const char *>(S.z) + (e >> 8));
                        uint64_t h = amj_hash_step(*reinterpret_cast<const uint64_t *>(
                                                       reinterpret_cast<const char *>(S.p) + zz.y + (e & 0xffu)),
                                                   zz.x);
                        if (zz.y) h = amj_hash_step(h, ida);
                        chk += h;
                        if (WRITE) {
                            int32_t v[4] = {ida, xid, S.yid[(e & 0xffu) >> 3], zz.x};   // a to its place
#pragma unroll
                            for (int k = 0; k < 3; k++)
                                if (v[k] > v[k + 1]) {
                                    const int32_t t = v[k];
                                    v[k] = v[k + 1];
                                    v[k + 1] = t;
                                }
                            if (pos < A.out_cap)
                                for (int k = 0; k < 4; k++) A.out[k][pos] = v[k];
                            pos += 32;
                        }
                    }
                    __syncwarp();
                }
                __syncwarp();
            }
        }
    }
    cnt = warp_sum(cnt);
    chk = warp_sum(chk);
    if ((threadIdx.x & 31) == 0 && cnt) {
        atomicAdd(A.count, cnt);
        atomicAdd(A.checksum, chk);
    }
}

// Transpose of a 32 x 32 bit block, row r in lane r.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t v, uint32_t lane) {
    uint32_t mask = 0x0000ffffu;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const uint32_t o = __shfl_xor_sync(AMJ_FULL_MASK, v, d);
        // lanes with bit d clear take the other lane's low columns into their high ones
        v = (lane & d) ? ((v & ~mask) | ((o & ~mask) >> d)) : ((v & mask) | ((o & mask) << d));
        mask ^= mask << (d >> 1);
    }
    return v;
}

// The wedge kernel leaves the edge between the children at places x < y as
// bit y of row x or as bit x of row y, whichever ranks lower: afterwards every
// row x has its bits y > x (bits below x are not read).  One warp a block row
// of 32 rows: block (i, k) takes in the transpose of block (k, i).
__global__ __launch_bounds__(256) void c4m_mirror_kernel(const TrieRef T, const int32_t *__restrict__ src1, uint64_t n,
                                                        const uint64_t *__restrict__ moff, uint32_t *mtx) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        const uint64_t j = base + lane;
        uint32_t deg = 0, row = 1;
        uint64_t mb = 0;
        if (j < n) {
            const int32_t a = src1[j];
            uint64_t ta, te;
            child_range(T, a, ta, te);
            deg = (uint32_t)(te - ta);
            row = (uint32_t)(j - ta);
            mb = moff[a];
        }
        unsigned todo = __ballot_sync(AMJ_FULL_MASK, (row & 31) == 0 && row + 1 < deg);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t d = __shfl_sync(AMJ_FULL_MASK, deg, l), r0 = __shfl_sync(AMJ_FULL_MASK, row, l);
            const uint32_t w = (d + 31) / 32, i = r0 / 32;
            uint32_t *M = mtx + __shfl_sync(AMJ_FULL_MASK, mb, l);
            for (uint32_t k = i; k < w; k++) {
                const uint32_t lo = 32 * k + lane < d ? M[(32 * k + lane) * w + i] : 0u;
                const uint32_t t = warp_transpose32(lo, lane);
                if (r0 + lane < d && t) M[(r0 + lane) * w + k] |= t;
            }
        }
    }
}

// Child lists of up to 32 E entries: their vertex ids in increasing order
// (sid), every entry's place in that order (pid), the place of a's own id.
template <int E>
__device__ __forceinline__ uint32_t c4m_order_row(const int32_t *__restrict__ data1, const int32_t *__restrict__ inv,
                                                  int32_t *sid, uint16_t *__restrict__ pid, uint64_t s, uint32_t len,
                                                  int32_t ida, uint32_t lane) {
    int32_t x[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const uint32_t i = e * 32u + lane;
        x[e] = i < len ? inv[data1[s + i]] : INT32_MAX;
    }
    uint32_t below = 0;
#pragma unroll
    for (int e = 0; e < E; e++) below += (e * 32u + lane < len && x[e] < ida) ? 1u : 0u;
    warp_bitonic_sort<E>(x, lane);
#pragma unroll
    for (int e = 0; e < E; e++)
        if (lane * E + e < len) sid[s + lane * E + e] = x[e];
    __syncwarp();
    for (uint32_t i = lane; i < len; i += 32) {
        const int32_t id = inv[data1[s + i]];
        uint32_t lo = 0, hi = len;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sid[s + mid] < id) lo = mid + 1;
            else hi = mid;
        }
        pid[s + i] = (uint16_t)lo;
    }
    return warp_sum(below);
}

__global__ __launch_bounds__(256, 4) void c4m_order_kernel(const TrieRef T, uint64_t nv, const int32_t *__restrict__ inv,
                                                          int32_t *sid, uint16_t *__restrict__ pid,
                                                          uint16_t *__restrict__ pa) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv; v += warps) {
        uint64_t s, e;
        child_range(T, (int32_t)v, s, e);
        const uint32_t len = (uint32_t)(e - s);
        if (!len) continue;
        const int32_t ida = inv[v];
        uint32_t below;
        if (len <= 32) below = c4m_order_row<1>(T.data1, inv, sid, pid, s, len, ida, lane);
        else if (len <= 64) below = c4m_order_row<2>(T.data1, inv, sid, pid, s, len, ida, lane);
        else if (len <= 128) below = c4m_order_row<4>(T.data1, inv, sid, pid, s, len, ida, lane);
        else if (len <= 256) below = c4m_order_row<8>(T.data1, inv, sid, pid, s, len, ida, lane);
        else if (len <= 512) below = c4m_order_row<16>(T.data1, inv, sid, pid, s, len, ida, lane);
        else below = c4m_order_row<32>(T.data1, inv, sid, pid, s, len, ida, lane);
        if (lane == 0) pa[v] = (uint16_t)below;
    }
}

int lftj_tri_matrices(amj_ctx *ctx, const Trie2 &R, const uint64_t *wedge, const uint16_t *pid, uint64_t nv,
                      uint32_t rank_bits, uint64_t max_words, DBuf<uint64_t> *moff, uint32_t **mtx, uint64_t *words);

// Largest child list of the trie (its longest out-neighbour list).
static int trie_max_children(amj_ctx *ctx, const Trie2 &T, uint64_t *maxc) {
    *maxc = 0;
    if (T.len0 == 0) return AMJ_OK;
    DBuf<unsigned long long> m;
    AMJ_TRY(m.alloc(ctx, 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(m.p, 0, sizeof(unsigned long long), ctx->stream));
    note_launch(ctx);
    max_children_kernel<<<(unsigned)std::min<uint64_t>((T.len0 + 255) / 256, (uint64_t)ctx->num_sms * 8), 256, 0,
                          ctx->stream>>>(T.off0.p, T.len0, m.p);
    AMJ_CUDA_TRY(cudaGetLastError());
    unsigned long long h = 0;
    AMJ_TRY(read_back(ctx, &h, m.p, sizeof(h)));
    *maxc = h;
    return AMJ_OK;
}

// Prepared state of the matrix path over one degree-ranked trie.
struct C4Matrix {
    DBuf<uint64_t> moff;
    uint32_t *mtx = nullptr;   // the context's matrix buffer
    DBuf<int32_t> sid;         // every child list by vertex id
    DBuf<uint16_t> pa;         // place of each rank's own id among its children's
};

// Whether the matrix path takes the degree-ranked trie T (every out-degree at
// most 1024, the matrices within half the free device memory), and if so the
// child lists by id and the triangle matrices.
int lftj_clique4_matrix_prepare(amj_ctx *ctx, const Trie2 &T, const int32_t *inv, const uint64_t *wedge, uint64_t nv,
                                uint32_t rank_bits, C4Matrix **out) {
    *out = nullptr;
    uint64_t maxc = 0;
    AMJ_TRY(trie_max_children(ctx, T, &maxc));
    if (maxc > C4M_MAX_DEG) return AMJ_OK;
    size_t fr = 0, tot = 0;
    AMJ_CUDA_TRY(cudaMemGetInfo(&fr, &tot));
    auto *m = new C4Matrix();
    uint64_t words = 0;
    // at most half the free memory, or the buffer the context already holds
    const uint64_t max_words = std::max<uint64_t>(fr / 2 / 4, ctx->c4_mtx_words);
    DBuf<uint16_t> pid;   // read in aligned groups of four, past the last entry
    int rc = m->sid.alloc(ctx, T.len1 ? T.len1 : 1);
    if (rc == AMJ_OK) rc = m->pa.alloc(ctx, nv ? nv : 1);
    if (rc == AMJ_OK) rc = pid.alloc(ctx, T.len1 + TRIE_LEVEL1_PAD);
    if (rc == AMJ_OK && T.len1) {
        note_launch(ctx);
        c4m_order_kernel<<<(unsigned)std::min<uint64_t>((nv * 32 + 255) / 256, (uint64_t)ctx->num_sms * 16), 256, 0,
                           ctx->stream>>>(trie_ref(T), nv, inv, m->sid.p, pid.p, m->pa.p);
        if (cudaGetLastError() != cudaSuccess) rc = fail(AMJ_ECUDA, "LFTJ 4-clique: child lists by id");
    }
    if (rc == AMJ_OK)
        rc = lftj_tri_matrices(ctx, T, wedge, pid.p, nv, rank_bits, max_words, &m->moff, &m->mtx, &words);
    if (rc == AMJ_OK && T.len1) {
        note_launch(ctx);
        c4m_mirror_kernel<<<(unsigned)std::min<uint64_t>((T.len1 + 255) / 256, (uint64_t)ctx->num_sms * 16), 256, 0,
                            ctx->stream>>>(trie_ref(T), T.src1.p, T.len1, m->moff.p, m->mtx);
        if (cudaGetLastError() != cudaSuccess) rc = fail(AMJ_ECUDA, "LFTJ 4-clique: mirrored matrices");
    }
    if (rc != AMJ_OK) {
        delete m;
        return rc == AMJ_ENOMEM ? AMJ_OK : rc;   // the matrices do not fit: not this path
    }
    *out = m;
    return AMJ_OK;
}

void lftj_clique4_matrix_release(C4Matrix *m) { delete m; }

// 4-cliques of the degree-ranked trie T from its prepared matrices: count and
// checksum, and with out the sorted tuples (out_cap rows available).
int lftj_clique4_matrix(amj_ctx *ctx, const Trie2 &T, const int32_t *inv, const C4Matrix *m, int32_t *const *out,
                        uint64_t out_cap, uint64_t *count, uint64_t *checksum, uint64_t *written, double *kernel_ms) {
    DBuf<C4Counters> ctr;
    AMJ_TRY(ctr.alloc(ctx, 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(ctr.p, 0, sizeof(C4Counters), ctx->stream));
    *count = *checksum = 0;
    if (written) *written = 0;
    if (T.len1 == 0) return AMJ_OK;
    const bool write = out != nullptr;
    C4MArgs A{};
    A.src1 = T.src1.p;
    A.inv = inv;
    A.sid = m->sid.p;
    A.pa = m->pa.p;
    A.T = trie_ref(T);
    A.moff = m->moff.p;
    A.mtx = m->mtx;
    A.n = T.len1;
    A.cursor = &ctr.p->cursor;
    A.count = &ctr.p->count;
    A.checksum = &ctr.p->checksum;
    A.out_cursor = &ctr.p->out_cursor;
    if (write) {
        for (int i = 0; i < 4; i++) A.out[i] = out[i];
        A.out_cap = out_cap;
    }
    auto kern = write ? lftj_clique4_matrix_kernel<true> : lftj_clique4_matrix_kernel<false>;
    int per_sm = 0;
    AMJ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C4M_THREADS, 0));
    if (per_sm < 1) per_sm = 1;
    AMJ_CUDA_TRY(cudaEventRecord(ctx->kev[0], ctx->stream));
    note_launch(ctx);
    kern<<<(unsigned)(ctx->num_sms * per_sm), C4M_THREADS, 0, ctx->stream>>>(A);
    AMJ_CUDA_TRY(cudaGetLastError());
    AMJ_CUDA_TRY(cudaEventRecord(ctx->kev[1], ctx->stream));
    C4Counters h;
    AMJ_TRY(read_back(ctx, &h, ctr.p, sizeof(h)));
    if (kernel_ms) *kernel_ms += event_ms(ctx->kev[0], ctx->kev[1]);
    *count = h.count;
    *checksum = h.checksum;
    if (written) *written = std::min<unsigned long long>(h.out_cursor, out_cap);
    return AMJ_OK;
}

int lftj_clique4(amj_ctx *ctx, const Trie2 &T, int32_t *const *out, uint64_t out_cap, uint64_t *count,
                 uint64_t *checksum, uint64_t *written, double *kernel_ms, int sorted_out) {
    DBuf<C4Counters> ctr;
    AMJ_TRY(ctr.alloc(ctx, 1));
    AMJ_CUDA_TRY(cudaMemsetAsync(ctr.p, 0, sizeof(C4Counters), ctx->stream));
    *count = *checksum = 0;
    if (written) *written = 0;
    if (T.len1 == 0) return AMJ_OK;
    // the longest child list bounds C(a,b): the size of every warp's scratch area
    note_launch(ctx);
    max_children_kernel<<<(unsigned)std::min<uint64_t>((T.len0 + 255) / 256, (uint64_t)ctx->num_sms * 8), 256, 0,
                          ctx->stream>>>(T.off0.p, T.len0, &ctr.p->max_deg);
    AMJ_CUDA_TRY(cudaGetLastError());
    unsigned long long max_deg = 0;
    AMJ_CUDA_TRY(cudaMemcpyAsync(&max_deg, &ctr.p->max_deg, 8, cudaMemcpyDeviceToHost, ctx->stream));
    AMJ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    const bool write = out != nullptr;
    auto kern = write ? lftj_clique4_kernel<true> : lftj_clique4_kernel<false>;
    int per_sm = 0;
    AMJ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0));
    uint64_t blocks = (uint64_t)ctx->num_sms * std::max(per_sm, 1);
    const uint64_t cap = std::max<unsigned long long>(max_deg, 1);
    // keep the scratch areas within 1/8 of the free device memory
    size_t fr = 0, tot = 0;
    AMJ_CUDA_TRY(cudaMemGetInfo(&fr, &tot));
    while (blocks > (uint64_t)ctx->num_sms && blocks * 8 * cap * 4 > fr / 8) blocks -= ctx->num_sms;
    if (blocks * 8 * cap * 4 > fr / 2) return fail(AMJ_ENOMEM, "LFTJ 4-clique: no room for the per-warp scratch");
    DBuf<int32_t> scratch;
    AMJ_TRY(scratch.alloc(ctx, blocks * 8 * cap));
    C4Args A{};
    A.src = T.src1.p;
    A.dst = T.data1.p;
    A.n = T.len1;
    A.T = trie_ref(T);
    A.cursor = &ctr.p->cursor;
    A.count = &ctr.p->count;
    A.checksum = &ctr.p->checksum;
    A.out_cursor = &ctr.p->out_cursor;
    if (write) {
        for (int i = 0; i < 4; i++) A.out[i] = out[i];
        A.out_cap = out_cap;
    }
    A.scratch = scratch.p;
    A.scratch_cap = cap;
    A.sorted_out = sorted_out;
    AMJ_CUDA_TRY(cudaEventRecord(ctx->kev[0], ctx->stream));
    note_launch(ctx);
    kern<<<(unsigned)blocks, 256, 0, ctx->stream>>>(A);
    AMJ_CUDA_TRY(cudaGetLastError());
    AMJ_CUDA_TRY(cudaEventRecord(ctx->kev[1], ctx->stream));
    C4Counters h;
    AMJ_CUDA_TRY(cudaMemcpyAsync(&h, ctr.p, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    AMJ_TRY(status_check(ctx, "LFTJ 4-clique"));
    if (kernel_ms) *kernel_ms += event_ms(ctx->kev[0], ctx->kev[1]);
    *count = h.count;
    *checksum = h.checksum;
    if (written) *written = std::min<unsigned long long>(h.out_cursor, out_cap);
    return AMJ_OK;
}

}  // namespace amj
