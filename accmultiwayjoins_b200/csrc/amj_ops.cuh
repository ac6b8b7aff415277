// Index structures and operator entry points shared between the translation
// units of libamj.
#pragma once
#include "amj_cuda.cuh"

struct ResultOwner {
    amj_ctx *ctx = nullptr;
    // pinned block of all host columns, back to the context's pool on release
    // (a result may outlive its context, whose pool then keeps no block)
    void *host_block = nullptr;
    std::shared_ptr<amj::ResultPool> host_pool;
    size_t host_bytes = 0;
};

namespace amj {

void result_init(amj_result *res, int k);

// Key of a hash index: the build relation's first column, or the pair of
// its first two columns (used when every column of the build relation is
// already bound at its level, i.e. the table only filters).
enum KeyMode : int { KEY_SINGLE = 0, KEY_PAIR = 1 };

constexpr int32_t OA_EMPTY_KEY = INT32_MIN;   // open addressing / cuckoo empty slot marker
constexpr int CUCKOO_SLOTS = 4;                // slots per cuckoo bucket (one 32-byte sector)

// A hash index over a build relation with at most 4 columns.  For the bucket
// layout the relation's columns are stored in bucket order next to each other
// (structure of arrays) so a probe reads the key and the bound payload from
// the same position: no row-id indirection into the original relation, unlike
// the reference's hash_keys / idx_in_origin / data[] triple
// (MHJ-GPU/Relation.cuh:50-63).  Open addressing and cuckoo store (c0, c1)
// pairs in 8-byte slots, four to a 32-byte sector.
struct HashIndex {
    int layout = AMJ_LAYOUT_BUCKET;
    int key_mode = KEY_SINGLE;
    uint64_t n = 0;
    int ncols = 0;
    uint32_t mask = 0;             // buckets-1, capacity-1, or cuckoo buckets-1
    DBuf<uint32_t> buc_ptrs;       // bucket layout: buckets+1 offsets
    DBuf<int32_t> cols[4];         // bucket layout: columns in bucket order
    DBuf<int2> slots;              // open addressing / cuckoo
    DBuf<char> block;              // memory of buc_ptrs and cols where a counting build laid them out together
};

// One index of build_bucket_indexes.
struct BucketSpec {
    const int32_t *cols[4];
    int ncols;
    uint64_t n;
    int key_mode;
    HashIndex *out;
};
constexpr uint64_t BUCKET_COUNT_MAX = 1ull << 23;   // rows of an index that the counting build takes
constexpr int BUCKET_BUILD_MAX = 8;                 // indexes of one build_bucket_indexes call
// Bucket indexes of up to BUCKET_COUNT_MAX rows each, all built by one set of
// launches in one block of memory, which `block` owns.  *zeroed (optional)
// gets BUCKET_ZEROED zeroed bytes of the block (null when count is 0).
constexpr size_t BUCKET_ZEROED = 64;
int build_bucket_indexes(amj_ctx *ctx, const BucketSpec *specs, int count, DBuf<char> *block, void **zeroed = nullptr);

int build_hash_index(amj_ctx *ctx, const int32_t *const *d_cols, int ncols, uint64_t n, int layout,
                     int key_mode, float load_factor, HashIndex *out);

// 2-level trie (CSR): level 0 distinct first-column values, offsets into
// level 1, level 1 second-column values sorted within each group.
struct Trie2 {
    uint64_t len0 = 0, len1 = 0;
    DBuf<int32_t> data0;
    DBuf<uint64_t> off0;
    DBuf<int32_t> data1;
    DBuf<int32_t> src1;        // level-0 value of every level-1 entry (sorted first column)
    DBuf<uint64_t> rowptr;     // dense child offsets for values rp_min .. rp_min+rp_count-1 (+1 end entry)
    int32_t rp_min = 0;
    uint64_t rp_count = 0;     // 0 when no dense array was built
    uint64_t range1 = 0;       // level 1's values span at most this many (0: not known)
};

// Level 1 of a trie of build_trie2 or build_trie2_ranked has TRIE_LEVEL1_PAD spare
// values after its last one, so kernels may read it in aligned 16-byte quads.
constexpr uint64_t TRIE_LEVEL1_PAD = 4;
// mm_known: least and greatest values of both columns with their signs flipped,
// where the caller has them;
// distinct: drop repeated rows (the set semantics of the leapfrog triejoin);
// vmax >= 0: every value of both columns lies in [0, vmax] (no min/max pass)
int build_trie2(amj_ctx *ctx, const int32_t *d_c0, const int32_t *d_c1, uint64_t n, Trie2 *out,
                bool distinct = false, int32_t vmax = -1, const uint32_t *mm_known = nullptr);
// The distinct 2-level tries of up to TRIE_JOBS_MAX relations, built together where
// their rows can be bucketed by counting (trie.cu), the others as build_trie2
// builds them.  `block` owns memory of the tries; level 0 of a trie built
// with others lists every value of the first column's range, and its level 1 may
// start at any value of an array: no aligned groups of four, no spare values.
constexpr int TRIE_JOBS_MAX = 3;
struct TrieCols {
    const int32_t *c0, *c1;
    uint64_t n;
};
int build_tries2(amj_ctx *ctx, const TrieCols *cols, int count, Trie2 *out, DBuf<char> *block);

// The distinct 2-level trie of the degree-ranked copy of the edges (c0, c1):
// every vertex renamed to its rank (below nv), edges from the lower to the
// higher rank.  Rows bucketed by counting, each row sorted on its own; the
// radix-sort build where a row is too long.  Level 0 holds every rank.
int build_trie2_ranked(amj_ctx *ctx, const int32_t *d_c0, const int32_t *d_c1, uint64_t n, const int32_t *rank,
                       uint64_t nv, Trie2 *out);

// time between two events recorded on the context stream (ms)
double event_ms(cudaEvent_t a, cudaEvent_t b);

// Degree-ordered copy (ns, nd) of the edge relation (c0, c1) when every edge
// has 0 <= c0 < c1 (*oriented); otherwise nothing is allocated.
int degree_ordered_copy(amj_ctx *ctx, const int32_t *c0, const int32_t *c1, uint64_t n, DBuf<int32_t> *ns,
                        DBuf<int32_t> *nd, bool *oriented);

// Ranks of the vertices in order of their degrees (about: degree_bin in
// graph_order.cu) when every edge has 0 <= c0 < c1 (*oriented): *rank[id] and
// *inv[rank] over ids 0..*nv-1.
int degree_ranks(amj_ctx *ctx, const int32_t *c0, const int32_t *c1, uint64_t n, DBuf<int32_t> *rank,
                 DBuf<int32_t> *inv, uint64_t *nv, bool *oriented);
// The level-1 entries of a degree-ranked trie grouped by b (a stable sort).
int build_wedges(amj_ctx *ctx, const Trie2 &R, uint64_t nv, DBuf<uint64_t> *out);

// copy materialised device result columns to pinned host memory (when asked)
int finish_result_columns(amj_ctx *ctx, amj_result *res, int flags);

}  // namespace amj

namespace amj {
constexpr int TRIE_MAX_LEVELS = 8;

// N-level trie: level l holds the last values of the distinct (l+1)-prefixes
// of the sorted rows, off[l] the offsets of their children in level l+1; the
// last level is the sorted last column, duplicates kept.
struct TrieN {
    int levels = 0;
    uint64_t len[TRIE_MAX_LEVELS] = {};
    DBuf<int32_t> data[TRIE_MAX_LEVELS];
    DBuf<uint64_t> off[TRIE_MAX_LEVELS - 1];
};

int build_trieN(amj_ctx *ctx, const int32_t *const *d_cols, int ncols, uint64_t n, TrieN *out);
}  // namespace amj

// A trie handle: a 2-level trie (t, levels = 0 in tn) or an N-level one (tn).
struct amj_trie {
    amj_ctx *ctx = nullptr;
    amj::Trie2 t;
    amj::TrieN tn;
    int levels() const { return tn.levels ? tn.levels : 2; }
    uint64_t len(int l) const { return tn.levels ? tn.len[l] : (l == 0 ? t.len0 : t.len1); }
    const int32_t *data(int l) const { return tn.levels ? tn.data[l].p : (l == 0 ? t.data0.p : t.data1.p); }
    const uint64_t *off(int l) const { return tn.levels ? tn.off[l].p : t.off0.p; }
};
