// AMHJ flat paths for star- and chain-shaped queries.
//
// When every build level is looked up by an attribute of the probe relation
// (a star: a fact table and its dimensions) and compares nothing but that
// key, the levels are independent: a probe row's result is the cross product
// of its matches in each level.  The frontier DFS (amhj_kernel.cuh) visits
// the levels one after another, so the latencies of a row's lookups add up.
// Here one thread takes one probe row, issues the bucket-bound loads of every
// level together, scans each (short) bucket for its key, and counts and
// hashes the product's tuples in attribute order.  A row whose product
// exceeds STAR_MAX_PRODUCT (a skewed dimension) is listed instead and joined
// afterwards by the DFS kernel, which shares such work across warps.
// Count mode only; bucket layout only.  Stars and chains in the numbering of
// the reference's benchmarks also have kernels over 16- and 32-byte bucket
// heads (amhj_star_canon_kernel, amhj_chain_canon_kernel, below), and
// materialised stars two flat passes (star_rowcount_kernel,
// star_write_kernel).
#pragma once
#include "amhj_probe.cuh"

namespace amj {

constexpr uint32_t STAR_MAX_PRODUCT = 256;

// whether plan P takes the flat path
inline bool star_eligible(const ProbePlan &P) {
    if (P.L < 1 || P.has_inl || P.sort_out || P.fib_level >= 0) return false;
    for (int l = 0; l < P.L; l++) {
        const LevelDesc &lv = P.lv[l];
        if (lv.layout != AMJ_LAYOUT_BUCKET || lv.key_mode != KEY_SINGLE || lv.cmp_mask != 1u) return false;
        bool from_probe = false;
        for (int c = 0; c < P.probe_ncols; c++) from_probe |= P.probe_attr[c] == lv.key_attr[0];
        if (!from_probe) return false;
    }
    return true;
}

// Totals of a flat kernel, and the rows it listed.
struct FlatCtr {
    unsigned long long count, checksum;
    unsigned int nover, done;   // listed rows; blocks that have ended
    unsigned int npair, pad;    // chain: listed matches
};

// A block's count and checksum added to the totals: one atomic a block, since
// the flat kernels run in many short blocks and the totals are two addresses
// (one a warp cost 0.3 ms at 37K blocks).  The last block writes the totals to
// pinned host memory, which saves the query a copy.  256-thread blocks.
__device__ __forceinline__ void flat_totals(unsigned long long cnt, unsigned long long chk, FlatCtr *ctr, FlatCtr *host) {
    __shared__ unsigned long long c[8], h[8];
    cnt = warp_sum(cnt);
    chk = warp_sum(chk);
    if ((threadIdx.x & 31) == 0) {
        c[threadIdx.x >> 5] = cnt;
        h[threadIdx.x >> 5] = chk;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; i++) {
            cnt += c[i];
            chk += h[i];
        }
        if (cnt) {
            atomicAdd(&ctr->count, cnt);
            atomicAdd(&ctr->checksum, chk);
        }
        __threadfence();
        if (atomicAdd(&ctr->done, 1u) == gridDim.x - 1) {
            __threadfence();   // the other blocks' sums before the reads below
            host->count = atomicAdd(&ctr->count, 0ull);
            host->checksum = atomicAdd(&ctr->checksum, 0ull);
            host->nover = atomicAdd(&ctr->nover, 0u);
            host->npair = atomicAdd(&ctr->npair, 0u);
            __threadfence_system();
        }
    }
}

__global__ __launch_bounds__(256) void amhj_star_kernel(const __grid_constant__ ProbePlan P,
                                                        FlatCtr *ctr, FlatCtr *host, uint32_t *over) {
    unsigned long long cnt = 0, chk = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = P.row_lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < P.row_hi; r += stride) {
        int32_t vals[AMJ_MAX_ATTRS];
        for (int c = 0; c < P.probe_ncols; c++) vals[P.probe_attr[c]] = P.probe_col[c][r];
        int32_t key[AMJ_MAX_BUILD_TABLES];
        uint32_t s[AMJ_MAX_BUILD_TABLES], e[AMJ_MAX_BUILD_TABLES];
        // every level's bucket bounds in flight together
#pragma unroll
        for (int l = 0; l < AMJ_MAX_BUILD_TABLES; l++) {
            if (l >= P.L) break;
            key[l] = vals[P.lv[l].key_attr[0]];
            const uint32_t h = (uint32_t)key[l] & P.lv[l].mask;
            s[l] = P.lv[l].buc_ptrs[h];
            e[l] = P.lv[l].buc_ptrs[h + 1];
        }
        uint32_t first[AMJ_MAX_BUILD_TABLES];
        uint64_t prod = 1;
#pragma unroll
        for (int l = 0; l < AMJ_MAX_BUILD_TABLES; l++) {
            if (l >= P.L) break;
            uint32_t nm = 0, f = e[l];
            for (uint32_t i = s[l]; i < e[l]; i++)
                if (P.lv[l].col[0][i] == key[l]) {
                    if (nm == 0) f = i;
                    nm++;
                }
            first[l] = f;
            prod *= nm;
        }
        if (prod == 0) continue;
        if (prod > STAR_MAX_PRODUCT) {
            over[atomicAdd(&ctr->nover, 1u)] = (uint32_t)(r - P.row_lo);
            continue;
        }
        if (prod == 1) {   // unique keys in every level: one tuple
#pragma unroll
            for (int l = 0; l < AMJ_MAX_BUILD_TABLES; l++) {
                if (l >= P.L) break;
                for (int c = 1; c < P.lv[l].ncols; c++) vals[P.lv[l].attr[c]] = P.lv[l].col[c][first[l]];
            }
            uint64_t h = AMJ_CHECKSUM_SEED;
            for (int a = 0; a < P.k; a++) h = amj_hash_step(h, vals[a]);
            cnt++;
            chk += h;
            continue;
        }
        // the product's tuples: one matching row per level, the last level fastest
        uint32_t pos[AMJ_MAX_BUILD_TABLES];
#pragma unroll
        for (int l = 0; l < AMJ_MAX_BUILD_TABLES; l++)
            if (l < P.L) pos[l] = first[l];
        while (true) {
#pragma unroll
            for (int l = 0; l < AMJ_MAX_BUILD_TABLES; l++) {
                if (l >= P.L) break;
                for (int c = 1; c < P.lv[l].ncols; c++) vals[P.lv[l].attr[c]] = P.lv[l].col[c][pos[l]];
            }
            uint64_t h = AMJ_CHECKSUM_SEED;
            for (int a = 0; a < P.k; a++) h = amj_hash_step(h, vals[a]);
            cnt++;
            chk += h;
            // next combination
            int l = P.L - 1;
            for (; l >= 0; l--) {
                uint32_t i = pos[l] + 1;
                while (i < e[l] && P.lv[l].col[0][i] != key[l]) i++;
                if (i < e[l]) {
                    pos[l] = i;
                    break;
                }
                pos[l] = first[l];
            }
            if (l < 0) break;
        }
    }
    flat_totals(cnt, chk, ctr, host);
}

// ---- the canonical star, count mode: one bucket head a lookup ----
// The shape of the reference's star benchmarks: probe F(0..L-1) and, for
// each key attribute c, one level D_c(c, L + c) of (key, payload) looked up
// by c.  The tuple is then (F's row, the payloads in key order), so every
// index below is a compile-time constant and the row's values stay in
// registers (the general kernel above indexes an attribute array at run time,
// a local-memory array, and loops over the levels).
//
// Before the probe every bucket of a level gets a head that holds its first
// rows (key, payload), so that a lookup is one load: the general kernel makes
// four per level (two bucket bounds, a key, a payload).  Dimension buckets
// hold one or two rows (keys unique, floorPow2(rows) buckets).  A row whose
// lookups each find one match in the heads is one tuple, hashed from the keys'
// shared prefix.  Other rows count their matches per level from the bounds and
// enumerate the product (an odometer over the levels, the last fastest);
// products above STAR_MAX_PRODUCT are listed for the DFS kernel as above.
// A star (star_canon) or chain (chain_canon) plan with its levels in key
// order: star level c is keyed by attribute c, chain level d by d + 1.
struct CanonPlan {
    const int32_t *fact[AMJ_MAX_BUILD_TABLES];     // probe columns (star: attribute c; chain: 0 and 1)
    const BucketHead *head[AMJ_MAX_BUILD_TABLES];  // bucket heads of level c
    const int32_t *key[AMJ_MAX_BUILD_TABLES];      // its key column
    const int32_t *pay[AMJ_MAX_BUILD_TABLES];      // its payload column (star: attribute L + c; chain: c + 2)
    const uint32_t *bp[AMJ_MAX_BUILD_TABLES];      // its bucket starts
    uint32_t nb[AMJ_MAX_BUILD_TABLES];             // its buckets (mask + 1)
    uint32_t mask[AMJ_MAX_BUILD_TABLES];
    uint64_t row_lo, row_hi;
};

// L when star plan P has the canonical shape (filling S but the heads), else 0
inline int star_canon(const ProbePlan &P, CanonPlan &S) {
    const int L = P.L;
    if (L < 1 || 2 * L > AMJ_MAX_ATTRS || P.probe_ncols != L || P.k != 2 * L) return 0;
    for (int c = 0; c < L; c++)
        if (P.probe_attr[c] != c) return 0;
    bool seen[AMJ_MAX_BUILD_TABLES] = {};
    for (int l = 0; l < L; l++) {
        const LevelDesc &lv = P.lv[l];
        const int c = lv.key_attr[0];
        if (c < 0 || c >= L || seen[c] || lv.ncols != 2 || lv.attr[0] != c || lv.attr[1] != L + c) return 0;
        seen[c] = true;
        S.fact[c] = P.probe_col[c];
        S.key[c] = lv.col[0];
        S.pay[c] = lv.col[1];
        S.bp[c] = lv.buc_ptrs;
        S.nb[c] = lv.mask + 1u;
        S.mask[c] = lv.mask;
    }
    S.row_lo = P.row_lo;
    S.row_hi = P.row_hi;
    return L;
}

struct HeadOut {
    BucketHead *p[AMJ_MAX_BUILD_TABLES];
};

// the heads of level blockIdx.y
__global__ void bucket_heads_kernel(const __grid_constant__ CanonPlan S, const __grid_constant__ HeadOut H) {
    const int c = blockIdx.y;
    const uint32_t nb = S.nb[c];
    const uint32_t *bp = S.bp[c];
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < nb; h += gridDim.x * blockDim.x) {
        BucketHead o;
        o.s = bp[h];
        o.e = bp[h + 1];
#pragma unroll
        for (int i = 0; i < HEAD_ROWS; i++) {
            const bool in = o.s + i < o.e;
            o.kp[2 * i] = in ? S.key[c][o.s + i] : 0;
            o.kp[2 * i + 1] = in ? S.pay[c][o.s + i] : 0;
        }
        H.p[c][h] = o;
    }
}

// A dimension bucket rarely holds more than two rows, and a lookup costs the L1
// by the bytes each lane loads (0.90 to 0.92 ms for 240 M lookups of 32-byte heads
// whatever the skew of the foreign keys, 1.11 ms as two 16-byte loads).  So the
// star reads 16-byte heads by one 128-bit load: two (key, payload) rows, of
// twice as many buckets (one more key bit), which take the same memory and
// overflow as rarely as three rows of a 32-byte head.  A free row holds a key
// of the neighbouring bucket, which no lookup here asks for; a bucket of more
// rows holds such keys with its index bucket's bounds as payloads, the first
// raised by one so that it is not zero.
// 60M-row star over 1M / 200K / 100K / 10K rows, Zipf(1.1) and uniform keys: 0.66
// and 0.81 ms (0.90 and 0.92 with 32-byte heads).
struct __align__(16) StarHead {
    int32_t k0, p0, k1, p1;
};
static_assert(sizeof(StarHead) == 16 && 2 * sizeof(StarHead) == sizeof(BucketHead), "two star heads a bucket");
// Blocks per SM: one lookup in flight a thread wants all of them (one dimension,
// 50M rows: 0.30 ms with four blocks, 0.20 with eight).  Two dimensions take five:
// rows with several matches run out of registers with more (4M rows, 8 matches in
// each: 2.49 ms with seven, 2.24 with five, 2.08 with four; one match in each, 8M
// rows: 0.197, 0.204 and 0.209).  16M rows of three dimensions with four, five, six
// and seven blocks: 0.361, 0.352, 0.347 and 0.380 ms; of four: 0.465, 0.451, 0.446,
// 0.596.
constexpr int star_blocks(int L) { return L == 1 ? 8 : L == 2 ? 5 : 6; }
// Dimensions up to which a row's overflowing buckets take their bounds from the
// heads (one dimension, 3 rows a key: 0.32 to 0.28 ms); with four, keeping the
// heads that long cost the rows with a key missing (0.32 to 0.37 ms).
constexpr int STAR_HEAD_BOUNDS = 2;
constexpr uint32_t STAR_HEAD_SCAN = 8;   // longer index buckets are taken as overflowing

// the heads of level blockIdx.y: index bucket h holds the rows of h and h + nb
__global__ void star_heads_kernel(const __grid_constant__ CanonPlan S, const __grid_constant__ HeadOut H) {
    const int c = blockIdx.y;
    const uint32_t nb = S.nb[c];
    const uint32_t *bp = S.bp[c];
    StarHead *out = reinterpret_cast<StarHead *>(H.p[c]);
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < nb; h += gridDim.x * blockDim.x) {
        const uint32_t s = bp[h], n = bp[h + 1] - s;
        // first of the two halves, then the other
        StarHead o[2];
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const int32_t none = (int32_t)((h + x * nb) ^ 1u);
            o[x] = StarHead{none, 0, none, 0};
            uint32_t m = 0;
            if (n <= STAR_HEAD_SCAN) {
                for (uint32_t i = 0; i < n; i++) {
                    const int32_t k = S.key[c][s + i];
                    if ((((uint32_t)k & nb) != 0) != (x != 0)) continue;
                    const int32_t p = S.pay[c][s + i];
                    if (m == 0) {
                        o[x].k0 = k;
                        o[x].p0 = p;
                    } else {
                        o[x].k1 = k;
                        o[x].p1 = p;
                    }
                    m++;
                }
            }
            if (n > STAR_HEAD_SCAN || m > 2) o[x] = StarHead{none, (int32_t)(s + 1), none, (int32_t)(s + n)};
            out[h + x * nb] = o[x];
        }
    }
}

template <int L>
__global__ __launch_bounds__(256, star_blocks(L)) void amhj_star_canon_kernel(const __grid_constant__ CanonPlan S,
                                                              FlatCtr *ctr, FlatCtr *host, uint32_t *over) {
    unsigned long long cnt = 0, chk = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = S.row_lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < S.row_hi; r += stride) {
        int32_t k[L];
#pragma unroll
        for (int c = 0; c < L; c++) k[c] = __ldcs(S.fact[c] + r);
        int4 w[L];
#pragma unroll
        for (int c = 0; c < L; c++)
            w[c] = __ldg(reinterpret_cast<const int4 *>(S.head[c]) + ((uint32_t)k[c] & (2 * S.nb[c] - 1)));
        bool one = true, empty = false;
        int32_t pay[L];
#pragma unroll
        for (int c = 0; c < L; c++) {
            const bool m0 = w[c].x == k[c], m1 = w[c].z == k[c];
            const uint32_t free_key = ((uint32_t)k[c] & (2 * S.nb[c] - 1)) ^ 1u;
            one &= m0 != m1;
            empty |= !m0 && !m1 && !((uint32_t)w[c].x == free_key && w[c].y != 0);
            pay[c] = m0 ? w[c].y : w[c].w;
        }
        if (empty) continue;   // a dimension without the key
        uint64_t hk = AMJ_CHECKSUM_SEED;
#pragma unroll
        for (int c = 0; c < L; c++) hk = amj_hash_step(hk, k[c]);
        if (one) {
            uint64_t h = hk;
#pragma unroll
            for (int c = 0; c < L; c++) h = amj_hash_step(h, pay[c]);
            cnt++;
            chk += h;
            continue;
        }
        uint32_t first[L], e[L];
        uint64_t prod = 1;
#pragma unroll
        for (int c = 0; c < L; c++) {
            const uint32_t b = (uint32_t)k[c] & S.mask[c];
            uint32_t s;
            if (L <= STAR_HEAD_BOUNDS && (uint32_t)w[c].x == (((uint32_t)k[c] & (2 * S.nb[c] - 1)) ^ 1u) && w[c].y != 0) {
                s = (uint32_t)w[c].y - 1;
                e[c] = (uint32_t)w[c].w;
            } else {
                s = S.bp[c][b];
                e[c] = S.bp[c][b + 1];
            }
            uint32_t nm = 0, f = e[c];
            for (uint32_t i = s; i < e[c]; i++)
                if (S.key[c][i] == k[c]) {
                    if (nm == 0) f = i;
                    nm++;
                }
            first[c] = f;
            prod *= nm;
        }
        if (prod == 0) continue;
        if (prod > STAR_MAX_PRODUCT) {
            over[atomicAdd(&ctr->nover, 1u)] = (uint32_t)(r - S.row_lo);
            continue;
        }
        uint32_t pos[L];
#pragma unroll
        for (int c = 0; c < L; c++) pos[c] = first[c];
        while (true) {
            uint64_t h = hk;
#pragma unroll
            for (int c = 0; c < L; c++) h = amj_hash_step(h, S.pay[c][pos[c]]);
            cnt++;
            chk += h;
            bool carry = true;
#pragma unroll
            for (int c = L - 1; c >= 0; c--) {
                if (carry) {
                    uint32_t i = pos[c] + 1;
                    while (i < e[c] && S.key[c][i] != k[c]) i++;
                    if (i < e[c]) {
                        pos[c] = i;
                        carry = false;
                    } else {
                        pos[c] = first[c];
                    }
                }
            }
            if (carry) break;
        }
    }
    flat_totals(cnt, chk, ctr, host);
}

// ---- the canonical chain, count mode: bucket rows handed out to lanes ----
// The shape of the reference's chain benchmarks: probe R0(0, 1) and levels
// R_d(d + 1, d + 2), level d looked up by the payload of level d - 1 (by
// attribute 1 at d = 0).  A warp looks up 32 probe rows, one a lane, stages the
// bucket heads (bounds and first rows) in shared memory and hands the buckets'
// rows out one a lane; with two levels the matches' buckets are handed out the
// same way, with more each lane walks its match's further levels depth first, a
// head a lookup.  The tuple hash is extended by one step a level, so a tuple
// costs one step at the last level.
// Bound by instructions: a walk of a probe row a lane kept 8.7 of 32 lanes
// active, since the rows' walks differ in length.  Measured, 3 x 1M rows,
// 14.6 M tuples: 165 us so, 126 with the first level handed out, 100 with
// both (and six blocks an SM).  Two or four matches a lane at a time, for more
// loads in flight: 129 and 164 us.
// A probe row whose first bucket, or a match whose further levels, hold more
// than CHAIN_ROW_BUDGET bucket rows (skewed keys) count nothing and are listed
// for the DFS kernel, which shares such work across warps.
constexpr uint32_t CHAIN_ROW_BUDGET = 128;

// L when plan P has the canonical chain shape (filling S but the heads), else 0
inline int chain_canon(const ProbePlan &P, CanonPlan &S) {
    const int L = P.L;
    if (L < 1 || L + 2 > AMJ_MAX_ATTRS || P.probe_ncols != 2 || P.k != L + 2) return 0;
    if (P.has_inl || P.sort_out || P.fib_level >= 0 || P.probe_attr[0] != 0 || P.probe_attr[1] != 1) return 0;
    for (int l = 0; l < L; l++) {
        const LevelDesc &lv = P.lv[l];
        const int d = lv.key_attr[0] - 1;
        if (d != l || lv.layout != AMJ_LAYOUT_BUCKET || lv.key_mode != KEY_SINGLE ||
            lv.cmp_mask != 1u || lv.ncols != 2 || lv.attr[0] != d + 1 || lv.attr[1] != d + 2)
            return 0;
        S.key[d] = lv.col[0];
        S.pay[d] = lv.col[1];
        S.bp[d] = lv.buc_ptrs;
        S.nb[d] = lv.mask + 1u;
        S.mask[d] = lv.mask;
    }
    S.fact[0] = P.probe_col[0];
    S.fact[1] = P.probe_col[1];
    S.row_lo = P.row_lo;
    S.row_hi = P.row_hi;
    return L;
}

// the matches of key at level D and, through them, the levels below; false
// when the walk ran out of budget
template <int D, int L>
__device__ __forceinline__ bool chain_walk(const CanonPlan &S, int32_t key, uint64_t h, unsigned long long &rc,
                                           unsigned long long &rchk, uint32_t &budget) {
    uint32_t w[8];
    load_head(S.head[D] + ((uint32_t)key & S.mask[D]), w);
    const uint32_t n = w[1] - w[0];
    if (n > budget) return false;
    budget -= n;
    for (uint32_t i = 0; i < n; i++) {
        int32_t k, v;
        if (i < (uint32_t)HEAD_ROWS) {
            k = (int32_t)(i == 0 ? w[2] : (i == 1 ? w[4] : w[6]));
            v = (int32_t)(i == 0 ? w[3] : (i == 1 ? w[5] : w[7]));
        } else {
            k = S.key[D][w[0] + i];
            v = S.pay[D][w[0] + i];
        }
        if (k != key) continue;
        const uint64_t hv = amj_hash_step(h, v);
        if constexpr (D == L - 1) {
            rc++;
            rchk += hv;
        } else {
            if (!chain_walk<D + 1, L>(S, v, hv, rc, rchk, budget)) return false;
        }
    }
    return true;
}

// rows of up to 32 buckets, waiting to be handed out
struct ChainStage {
    unsigned long long hv[32];           // hash of the partial tuple
    int4 ent[32];                        // rows before the bucket's, bucket start, key, probe row
    int2 kp[HEAD_ROWS][32];              // the bucket's first rows
};

// The whole warp: lane's bucket of level d (head w, n rows, possibly none) was
// looked up by `key` from a partial tuple of hash hv; f(hit, row, payload, hash)
// is called by all lanes together, a bucket row a lane.
template <class F>
__device__ __forceinline__ void chain_spread(const CanonPlan &S, int d, ChainStage &W, int lane, uint32_t n,
                                             const uint32_t (&w)[8], int32_t key, unsigned long long hv, uint32_t row,
                                             F &&f) {
    const unsigned lt = lanemask_lt(), le = lt | (1u << lane);
    const uint32_t incl = warp_inclusive_scan(n, lane), excl = incl - n;
    const uint32_t tot = __shfl_sync(AMJ_FULL_MASK, incl, 31);
    const unsigned live = __ballot_sync(AMJ_FULL_MASK, n > 0);
    if (n) {
        const int at = __popc(live & lt);
        W.hv[at] = hv;
        W.ent[at] = make_int4((int)excl, (int)w[0], key, (int)row);
#pragma unroll
        for (int i = 0; i < HEAD_ROWS; i++) W.kp[i][at] = make_int2((int)w[2 + 2 * i], (int)w[3 + 2 * i]);
    }
    __syncwarp();
    int before = -1;   // buckets begun before this step, minus one
    for (uint32_t j0 = 0; j0 < tot; j0 += 32) {
        const unsigned begun = __reduce_or_sync(AMJ_FULL_MASK, n && excl - j0 < 32u ? 1u << (excl - j0) : 0u);
        const int o = before + __popc(begun & le);
        before += __popc(begun);
        const uint32_t j = j0 + lane;
        int2 kv = make_int2(0, 0);
        int4 e = make_int4(0, 0, 1, 0);
        if (j < tot) {
            e = W.ent[o];
            const uint32_t i = j - (uint32_t)e.x;
            if (i < (uint32_t)HEAD_ROWS) kv = W.kp[i][o];
            else kv = make_int2(S.key[d][(uint32_t)e.y + i], S.pay[d][(uint32_t)e.y + i]);
        }
        const bool hit = j < tot && kv.x == e.z;
        f(hit, (uint32_t)e.w, kv.y, hit ? amj_hash_step(W.hv[o], kv.y) : 0ull);
    }
    __syncwarp();
}

// six blocks per SM (40 registers) up to two levels (1M rows: 100 us; four blocks
// 116, eight 120), four (64 registers) at three (0.332 ms; 0.360 with six, 0.369
// with three); deeper walks keep their per-level state in two blocks' worth of
// registers (1M rows, four and five levels: 1.10 and 3.71 ms; three blocks measure
// 0.83 and 2.90, four 0.73 and 3.40)
template <int L>
__global__ __launch_bounds__(256, L <= 2 ? 6 : L <= 3 ? 4 : 2) void amhj_chain_canon_kernel(
    const __grid_constant__ CanonPlan S, FlatCtr *ctr, FlatCtr *host, uint32_t *over, uint2 *pairs,
    uint32_t pair_cap) {
    __shared__ ChainStage smem[L == 2 ? 2 : 1][8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long cnt = 0, chk = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    // a match whose walk is too long for a lane
    auto list = [&](uint32_t row, int32_t v) {
        if (*(volatile unsigned int *)&ctr->npair > pair_cap) return;   // so that the count cannot wrap
        const uint32_t at = atomicAdd(&ctr->npair, 1u);
        if (at < pair_cap) pairs[at] = make_uint2(row, (uint32_t)v);
    };
    for (uint64_t base = S.row_lo + blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); base < S.row_hi;
         base += stride) {
        const uint64_t r = base + lane;
        uint32_t n = 0, w[8] = {};
        int32_t a0 = 0, a1 = 0;
        if (r < S.row_hi) {
            a0 = __ldcs(S.fact[0] + r);
            a1 = __ldcs(S.fact[1] + r);
            load_head(S.head[0] + ((uint32_t)a1 & S.mask[0]), w);
            n = w[1] - w[0];
            if (n > CHAIN_ROW_BUDGET) {
                over[atomicAdd(&ctr->nover, 1u)] = (uint32_t)(r - S.row_lo);
                n = 0;
            }
        }
        chain_spread(S, 0, smem[0][wid], lane, n, w, a1, amj_hash_step(amj_hash_step(AMJ_CHECKSUM_SEED, a0), a1),
                     (uint32_t)(r - S.row_lo), [&](bool hit, uint32_t row, int32_t v, unsigned long long h) {
            if constexpr (L == 1) {
                cnt += hit;
                chk += h;
            } else if constexpr (L == 2) {
                uint32_t n1 = 0, w1[8] = {};
                if (hit) {
                    load_head(S.head[1] + ((uint32_t)v & S.mask[1]), w1);
                    n1 = w1[1] - w1[0];
                    if (n1 > CHAIN_ROW_BUDGET) {
                        list(row, v);
                        n1 = 0;
                    }
                }
                chain_spread(S, 1, smem[1][wid], lane, n1, w1, v, h, 0,
                             [&](bool hit1, uint32_t, int32_t, unsigned long long h1) {
                    cnt += hit1;
                    chk += h1;
                });
            } else if (hit) {
                unsigned long long rc = 0, rchk = 0;
                uint32_t budget = CHAIN_ROW_BUDGET;
                if (chain_walk<1, L>(S, v, h, rc, rchk, budget)) {
                    cnt += rc;
                    chk += rchk;
                } else {
                    list(row, v);
                }
            }
        });
    }
    flat_totals(cnt, chk, ctr, host);
}

// the listed matches as a probe relation (0, 1, 2) of the remaining levels
__global__ void chain_gather_kernel(const __grid_constant__ CanonPlan S, const uint2 *__restrict__ pairs, uint32_t n,
                                    int32_t *__restrict__ c0, int32_t *__restrict__ c1, int32_t *__restrict__ c2) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 p = pairs[i];
        c0[i] = S.fact[0][S.row_lo + p.x];
        c1[i] = S.fact[1][S.row_lo + p.x];
        c2[i] = (int32_t)p.y;
    }
}

// ---- materialised star joins (two flat passes) ----
// Pass 1: every probe row's number of result tuples (the product of its
// matches per level).  A scan turns them into output offsets.  Pass 2: every
// row writes its product's tuples from its offset, the last level fastest,
// and adds them to the count and checksum.  A row's tuples are written by
// its own thread, so the pass suits plans whose rows have few matches (the
// 2-relation parts of a staged join, stars over dimensions with unique
// keys); rows are independent, so the result is exact for any product.
__global__ __launch_bounds__(256) void star_rowcount_kernel(const __grid_constant__ ProbePlan P,
                                                            unsigned long long *__restrict__ rc) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = P.row_lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < P.row_hi; r += stride) {
        int32_t vals[AMJ_MAX_ATTRS];
        for (int c = 0; c < P.probe_ncols; c++) vals[P.probe_attr[c]] = P.probe_col[c][r];
        unsigned long long prod = 1;
        for (int l = 0; l < P.L && prod; l++) {
            const int32_t key = vals[P.lv[l].key_attr[0]];
            const uint32_t h = (uint32_t)key & P.lv[l].mask;
            const uint32_t s = P.lv[l].buc_ptrs[h], e = P.lv[l].buc_ptrs[h + 1];
            uint32_t nm = 0;
            for (uint32_t i = s; i < e; i++) nm += P.lv[l].col[0][i] == key;
            prod *= nm;
        }
        rc[r - P.row_lo] = prod;
    }
}

__global__ __launch_bounds__(256) void star_write_kernel(const __grid_constant__ ProbePlan P,
                                                         const unsigned long long *__restrict__ off,
                                                         unsigned long long *count, unsigned long long *checksum) {
    unsigned long long cnt = 0, chk = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = P.row_lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < P.row_hi; r += stride) {
        unsigned long long at = off[r - P.row_lo];
        if (off[r - P.row_lo + 1] == at) continue;   // no tuples
        int32_t vals[AMJ_MAX_ATTRS];
        for (int c = 0; c < P.probe_ncols; c++) vals[P.probe_attr[c]] = P.probe_col[c][r];
        int32_t key[AMJ_MAX_BUILD_TABLES];
        uint32_t first[AMJ_MAX_BUILD_TABLES], pos[AMJ_MAX_BUILD_TABLES], e[AMJ_MAX_BUILD_TABLES];
        for (int l = 0; l < P.L; l++) {
            key[l] = vals[P.lv[l].key_attr[0]];
            const uint32_t h = (uint32_t)key[l] & P.lv[l].mask;
            uint32_t i = P.lv[l].buc_ptrs[h];
            e[l] = P.lv[l].buc_ptrs[h + 1];
            while (P.lv[l].col[0][i] != key[l]) i++;   // a match exists: the row has tuples
            first[l] = pos[l] = i;
        }
        while (true) {
            for (int l = 0; l < P.L; l++)
                for (int c = 1; c < P.lv[l].ncols; c++) vals[P.lv[l].attr[c]] = P.lv[l].col[c][pos[l]];
            uint64_t hsh = AMJ_CHECKSUM_SEED;
            for (int a = 0; a < P.k; a++) {
                hsh = amj_hash_step(hsh, vals[a]);
                P.out[a][at] = vals[a];
            }
            at++;
            cnt++;
            chk += hsh;
            int l = P.L - 1;
            for (; l >= 0; l--) {
                uint32_t i = pos[l] + 1;
                while (i < e[l] && P.lv[l].col[0][i] != key[l]) i++;
                if (i < e[l]) {
                    pos[l] = i;
                    break;
                }
                pos[l] = first[l];
            }
            if (l < 0) break;
        }
    }
    cnt = warp_sum(cnt);
    chk = warp_sum(chk);
    if ((threadIdx.x & 31) == 0 && cnt) {
        atomicAdd(count, cnt);
        atomicAdd(checksum, chk);
    }
}

// the probe columns of the listed rows (row ids relative to row_lo)
__global__ void star_gather_kernel(const __grid_constant__ ProbePlan P, const uint32_t *rows, uint32_t n,
                                   int32_t *const *out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int c = 0; c < P.probe_ncols; c++) out[c][i] = P.probe_col[c][P.row_lo + rows[i]];
}

}  // namespace amj

namespace amj {

// ---- thread-per-row baseline ----
// The reference's MHJ (MHJ-GPU/Joins/MHJ.cuh:18-122): one thread per probe
// row walks the build levels depth first with backtracking, scanning each
// bucket alone.  Kept as a comparator for the warp-cooperative frontier DFS
// (AMJ_F_THREAD_PER_ROW); bucket layout, count mode.
inline bool thread_row_eligible(const ProbePlan &P) {
    if (P.L < 1 || P.fib_level >= 0) return false;
    for (int l = 0; l < P.L; l++)
        if (P.lv[l].layout != AMJ_LAYOUT_BUCKET) return false;
    return true;
}

__device__ __forceinline__ void thread_row_range(const LevelDesc &lv, const int32_t *vals, uint32_t &s, uint32_t &e) {
    const int32_t k0 = vals[lv.key_attr[0]];
    const uint32_t h = (lv.key_mode == KEY_PAIR ? hash_pair(k0, vals[lv.key_attr[1]]) : (uint32_t)k0) & lv.mask;
    s = lv.buc_ptrs[h];
    e = lv.buc_ptrs[h + 1];
}

__global__ __launch_bounds__(256) void amhj_thread_row_kernel(const __grid_constant__ ProbePlan P,
                                                              unsigned long long *count,
                                                              unsigned long long *checksum) {
    unsigned long long cnt = 0, chk = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = P.row_lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < P.row_hi; r += stride) {
        int32_t vals[AMJ_MAX_ATTRS];
        for (int c = 0; c < P.probe_ncols; c++) vals[P.probe_attr[c]] = P.probe_col[c][r];
        uint32_t pos[AMJ_MAX_BUILD_TABLES], end[AMJ_MAX_BUILD_TABLES];
        int d = 0;
        thread_row_range(P.lv[0], vals, pos[0], end[0]);
        while (true) {
            if (pos[d] >= end[d]) {
                if (d == 0) break;
                d--;
                pos[d]++;
                continue;
            }
            const LevelDesc &lv = P.lv[d];
            const uint32_t i = pos[d];
            bool ok = true;
            for (int c = 0; c < lv.ncols && ok; c++)
                if ((lv.cmp_mask >> c) & 1u) ok = lv.col[c][i] == vals[lv.attr[c]];
            if (!ok) {
                pos[d]++;
                continue;
            }
            for (int c = 0; c < lv.ncols; c++)
                if ((lv.bind_mask >> c) & 1u) vals[lv.attr[c]] = lv.col[c][i];
            if (d == P.L - 1) {
                int32_t t[AMJ_MAX_ATTRS];
                for (int a = 0; a < P.k; a++) t[a] = vals[a];
                if (P.sort_out)   // a degree-ordered copy reports every tuple sorted
                    for (int a = 1; a < P.k; a++)
                        for (int b = a; b > 0 && t[b - 1] > t[b]; b--) {
                            const int32_t x = t[b - 1];
                            t[b - 1] = t[b];
                            t[b] = x;
                        }
                uint64_t h = AMJ_CHECKSUM_SEED;
                for (int a = 0; a < P.k; a++) h = amj_hash_step(h, t[a]);
                cnt++;
                chk += h;
                pos[d]++;
                continue;
            }
            d++;
            thread_row_range(P.lv[d], vals, pos[d], end[d]);
        }
    }
    cnt = warp_sum(cnt);
    chk = warp_sum(chk);
    if ((threadIdx.x & 31) == 0 && cnt) {
        atomicAdd(count, cnt);
        atomicAdd(checksum, chk);
    }
}

}  // namespace amj
