"""Batched AMHJ (amj_batch_*): every query of a heterogeneous mix gives the
same count and checksum in the batch as alone (one query per call) and as the
oracle, for each layout, block size, task size, with and without a captured
CUDA graph; a replayed graph reads changed relation contents; the autotuner
returns a grid point."""
import numpy as np
import pytest

from accmultiwayjoins_b200 import AmjError, Context, _lib as L, data
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def oracle_of(q):
    if q["qt"] == "TRI":
        s, d = q["rels"][0][0]
        return O.triangle(s, d)
    return O.mhj(q["rels"])


@pytest.fixture(scope="module")
def mix():
    qs = list(data.query_mix(48, seed=7, min_rows=1000, max_rows=60000, out_cap=1 << 20))
    return qs, [oracle_of(q) for q in qs]


def submit_all(ctx, b, qs):
    keep = []
    for q in qs:
        rels = [ctx.relation(c, a) for c, a in q["rels"]]
        keep.append(rels)
        b.submit(q["qt"], rels)
    return keep


@pytest.mark.parametrize("layout", ["bucket", "oa"])
@pytest.mark.parametrize("block_size,task_chunk,load_factor", [(256, 1024, 0.0), (128, 32, 0.5), (512, 256, 0.85)])
def test_batch_matches_oracle(mix, layout, block_size, task_chunk, load_factor):
    qs, want = mix
    with Context(0) as ctx:
        b = ctx.batch()
        submit_all(ctx, b, qs)
        r = b.run(layout=layout, block_size=block_size, task_chunk=task_chunk, load_factor=load_factor)
        assert list(zip(r.counts, r.checksums)) == want
        assert r.tasks_popped == r.tasks_pushed
        assert r.units > 0 and r.launches > 0 and not r.graph


def test_batch_equals_one_query_per_call(mix):
    qs, want = mix
    with Context(0) as ctx:
        b = ctx.batch()
        keep = submit_all(ctx, b, qs)
        r = b.run()
        for q, rels, c, k in zip(qs, keep, r.counts, r.checksums):
            alone = ctx.amhj(q["qt"], rels)
            assert (alone.count, alone.checksum) == (c, k)


def test_batch_graph_capture_and_replay_reads_new_contents():
    import torch
    qs0 = list(data.query_mix(24, seed=11, min_rows=1000, max_rows=30000, out_cap=1 << 20))
    qs1 = list(data.query_mix(24, seed=11, min_rows=1000, max_rows=30000, out_cap=1 << 20))
    # same shapes and sizes, new contents: regenerate every column with another seed
    for q in qs1:
        for cols, _ in q["rels"]:
            for i, c in enumerate(cols):
                cols[i] = data.uniform(c.shape[0], 0, max(int(c.max()) + 1, 2), 99, i) if c.shape[0] else c
    with Context(0) as ctx:
        tensors = [[torch.from_numpy(c.copy()).cuda() for c in cols] for q in qs0 for cols, _ in q["rels"]]
        b = ctx.batch()
        it = iter(tensors)
        for q in qs0:
            rels = [ctx.relation(next(it), a) for _, a in q["rels"]]
            b.submit(q["qt"], rels)
        first = b.run(use_graph=True)
        again = b.run(use_graph=True)
        assert first.graph and again.graph
        want0 = [oracle_of(q) for q in qs0]
        assert list(zip(first.counts, first.checksums)) == want0
        assert list(zip(again.counts, again.checksums)) == want0
        # overwrite the borrowed device columns in place and replay
        new_cols = [cols for q in qs1 for cols, _ in q["rels"]]
        for ts, cols in zip(tensors, new_cols):
            for t, c in zip(ts, cols):
                t.copy_(torch.from_numpy(c))
        torch.cuda.synchronize()
        third = b.run(use_graph=True)
        assert list(zip(third.counts, third.checksums)) == [oracle_of(q) for q in qs1]
        eager = b.run(use_graph=False)
        assert (eager.counts, eager.checksums) == (third.counts, third.checksums)


def test_batch_work_sharing_across_queries():
    """Two skewed chains whose level-1 buckets are large, next to small
    queries: small tasks are pushed and popped across query boundaries."""
    q = [([data.uniform(100, 0, 100, 1), data.uniform(100, 0, 100, 2)], [0, 1]),
         ([data.uniform(2000, 0, 100, 3), data.uniform(2000, 0, 4, 4)], [1, 2]),
         ([data.uniform(20000, 0, 4, 5), data.uniform(20000, 0, 1 << 20, 6)], [2, 3])]
    small = data.chain_relations(3000, 1 << 12, 3, seed=5)
    want = [O.mhj(q), O.mhj(small), O.mhj(q)]
    with Context(0) as ctx:
        b = ctx.batch()
        for rels in (q, small, q):
            b.submit("NORMAL", [ctx.relation(c, a) for c, a in rels])
        r = b.run(task_chunk=32)
        assert list(zip(r.counts, r.checksums)) == want
        assert r.tasks_pushed > 0 and r.tasks_popped == r.tasks_pushed


@pytest.mark.parametrize("layout", ["bucket", "oa"])
def test_batch_limits_and_empty_relations(layout):
    """A 7-relation chain (6 build tables, 8 attributes), a 5-relation star,
    an empty build relation, an empty probe relation and a one-row query, in
    one batch: equal to one call per query and to the oracle."""
    long_chain = data.chain_relations(3000, 3000, 7, seed=31)
    fact, dims = data.star_relations(5000, [300, 200, 100, 50], theta=1.2, seed=32)
    star = [fact] + dims
    empty_build = data.chain_relations(2000, 256, 3, seed=33)
    empty_build[1] = ([np.zeros(0, np.int32), np.zeros(0, np.int32)], [1, 2])
    empty_probe = data.chain_relations(2000, 256, 3, seed=34)
    empty_probe[0] = ([np.zeros(0, np.int32), np.zeros(0, np.int32)], [0, 1])
    one = [([np.array([5], np.int32), np.array([7], np.int32)], [0, 1]),
           ([np.array([7, 7], np.int32), np.array([1, 2], np.int32)], [1, 2])]
    queries = [long_chain, star, empty_build, empty_probe, one]
    with Context(0) as ctx:
        b = ctx.batch()
        rels = []
        for q in queries:
            r = [ctx.relation(c, a) for c, a in q]
            rels.append(r)
            b.submit("NORMAL", r)
        got = b.run(layout=layout, block_size=256)
        for q, r, c, k in zip(queries, rels, got.counts, got.checksums):
            alone = ctx.amhj("NORMAL", r)
            assert (alone.count, alone.checksum) == (c, k) == O.mhj(q)
        assert got.counts[2] == 0 and got.counts[3] == 0 and got.counts[4] == 2


def test_batch_tuner_picks_a_grid_point(mix):
    qs, want = mix
    with Context(0) as ctx:
        b = ctx.batch()
        submit_all(ctx, b, qs)
        best, ms = b.tune(sample_every=4, load_factors=(0.5, 0.85), block_sizes=(128, 256), task_chunks=(64, 1024))
        assert best.load_factor in (np.float32(0.5), np.float32(0.85))
        assert best.block_size in (128, 256) and best.task_chunk in (64, 1024)
        assert ms > 0
        r = b.run(opts=best)
        assert list(zip(r.counts, r.checksums)) == want


def test_batch_rejects_what_it_does_not_run():
    with Context(0) as ctx:
        b = ctx.batch()
        with pytest.raises(AmjError) as e:
            b.run()
        assert e.value.status == L.AMJ_EINVAL
        one = ctx.relation([data.uniform(10, 0, 5, 1)], [0])
        with pytest.raises(AmjError) as e:
            b.submit("NORMAL", [one])
        assert e.value.status == L.AMJ_EUNSUPPORTED
        rels = [ctx.relation(c, a) for c, a in data.chain_relations(100, 50, 2, seed=1)]
        assert b.submit("NORMAL", rels) == 0
        with pytest.raises(AmjError) as e:
            b.run(block_size=96)
        assert e.value.status == L.AMJ_EINVAL
        r = b.run()
        assert (r.counts[0], r.checksums[0]) == O.mhj(data.chain_relations(100, 50, 2, seed=1))


def tri_edges(kind, n, seed):
    """Edge relations where one side's lists are much longer than the other's."""
    rng = np.random.default_rng(seed)
    if kind == "empty":
        return np.zeros(0, np.int32), np.zeros(0, np.int32)
    if kind == "hub_source":      # the hubs are first: long lists of a
        s, d = data.rmat(9, n, 0.57, 0.19, 0.19, seed)
    elif kind == "hub_target":    # the hubs are last: long lists of b
        s, d = data.rmat(9, n, 0.57, 0.19, 0.19, seed)
        s, d = 1000 - d, 1000 - s
    elif kind == "bag":           # any direction, self-loops, repeated rows, negative ids
        s = rng.integers(-20, 20, n).astype(np.int32)
        d = rng.integers(-20, 20, n).astype(np.int32)
    else:                         # sparse ids far above the bucket count, and few buckets hit
        s = (rng.integers(0, 60, n) * 65536 + 7).astype(np.int32)
        d = (rng.integers(0, 60, n) * 65536 + 7).astype(np.int32)
    return np.ascontiguousarray(s, np.int32), np.ascontiguousarray(d, np.int32)


@pytest.mark.parametrize("kind", ["empty", "hub_source", "hub_target", "bag", "sparse"])
@pytest.mark.parametrize("n", [1, 31, 33, 700, 5000])
def test_batch_triangle_queries(kind, n):
    """Triangle queries beside another one: the candidates of each edge come
    from the shorter list, repeated rows multiply, eager and replayed."""
    edges = [tri_edges(kind, n, s) for s in (1, 2)]
    want = [O.triangle(s, d) for s, d in edges]
    star = [([data.uniform(100, 0, 50, 1)], [0]), ([data.permutation(50, 2), data.uniform(50, 0, 9, 3)], [0, 1])]
    with Context(0) as ctx, ctx.batch() as b:
        for s, d in edges:
            b.submit("TRI", [ctx.relation([s, d], [0, 1])])
        b.submit("NORMAL", [ctx.relation(c, a) for c, a in star])
        want.append(O.mhj(star) if len(star) > 2 else (100, None))
        for graph in (False, True, True):
            r = b.run(use_graph=graph)
            assert list(zip(r.counts, r.checksums))[:2] == want[:2]
            assert r.counts[2] == 100


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, (1 << 23) - 5, (1 << 23) + 1])
def test_batch_index_builds_around_the_limits(n):
    """Index builds at the edges of a tile of rows and on both sides of the
    counting build's largest table, next to small tables of three columns."""
    small = [([data.uniform(300, 0, 40, 1), data.uniform(300, 0, 9, 2)], [0, 1]),
             ([data.uniform(500, 0, 9, 3), data.uniform(500, 0, 40, 4), data.uniform(500, 0, 99, 5)], [1, 0, 2])]
    big = [([data.uniform(4000, 0, 1 << 20, 6), data.uniform(4000, 0, max(n, 2), 7)], [0, 1]),
           ([data.uniform(n, 0, max(n, 2), 8), data.uniform(n, 0, 99, 9)], [1, 2])]
    with Context(0) as ctx, ctx.batch() as b:
        alone = []
        for q in (small, big, small):
            rels = [ctx.relation(c, a) for c, a in q]
            b.submit("NORMAL", rels)
            r = ctx.amhj("NORMAL", rels, plan="frontier")
            alone.append((r.count, r.checksum))
        r = b.run()
        assert list(zip(r.counts, r.checksums)) == alone
        assert alone[0] == alone[2] == O.mhj(small)
        if n < 1 << 20:
            assert alone[1] == O.mhj(big)


def test_batch_triangle_filter_of_a_long_bucket():
    """A triangle query with one edge repeated two million times: the pass
    that makes the filter's words does not read such a bucket row by row
    (170 ms of one thread, against a fraction of a millisecond)."""
    s, d = data.rmat(10, 8000, 0.57, 0.19, 0.19, 3)
    want = O.triangle(s, d)
    n = 2_000_000
    s, d = np.concatenate([s, np.full(n, 1024, np.int32)]), np.concatenate([d, np.full(n, 1025, np.int32)])
    with Context(0) as ctx, ctx.batch() as b:
        b.submit("TRI", [ctx.relation([s, d], [0, 1])])
        runs = [b.run(use_graph=True) for _ in range(4)]
        assert all((r.counts[0], r.checksums[0]) == want for r in runs)
        assert min(r.build_ms for r in runs) < 30.0


@pytest.mark.parametrize("copies", [1, 3, 63, 64, 65, 300])
def test_batch_triangles_through_repeated_edges(copies):
    """Buckets of the pair index as long as, and longer than, the rows that a
    filter word is made of: every copy of the closing edge counts."""
    s, d = data.rmat(8, 900, 0.57, 0.19, 0.19, copies)
    keep = np.arange(len(s)) % 7 == 0
    s = np.concatenate([s, np.repeat(s[keep], copies - 1)])
    d = np.concatenate([d, np.repeat(d[keep], copies - 1)])
    with Context(0) as ctx, ctx.batch() as b:
        b.submit("TRI", [ctx.relation([s, d], [0, 1])])
        r = b.run()
        assert (r.counts[0], r.checksums[0]) == O.triangle(s, d)


def test_batch_units_of_queries_without_a_second_frontier():
    """Triangles over open addressing end at their first level (the filter is
    inline): their units shrink to give each warp a few of them, not the many
    that even out the trees below a chain's level 0."""
    s, d = data.rmat(12, 1 << 16, 0.57, 0.19, 0.19, 5)
    chain = data.chain_relations(20_000, 1 << 12, 3, seed=2)
    with Context(0) as ctx, ctx.batch() as b:
        b.submit("TRI", [ctx.relation([s, d], [0, 1])])
        flat = b.run(layout="oa")
        assert (flat.counts[0], flat.checksums[0]) == O.triangle(s, d)
        assert 4000 <= flat.units <= 8 * 148 * 32 + 1   # with 64 a warp over 100 thousand
        b.submit("NORMAL", [ctx.relation(c, a) for c, a in chain])
        both = b.run(layout="oa")
        assert both.units - flat.units > 1000
        assert list(zip(both.counts, both.checksums)) == [(flat.counts[0], flat.checksums[0]), O.mhj(chain)]


@pytest.mark.parametrize("beside", ["nothing", "star", "chain"])
def test_batch_triangles_beside_other_queries(beside):
    """Triangle queries alone, and beside a query of the other kernel: every
    count and checksum, eager and replayed."""
    edges = [data.rmat(9, 3000, 0.57, 0.19, 0.19, s) for s in (1, 2, 3)]
    queries = [("TRI", [(list(e), [0, 1])], O.triangle(*e)) for e in edges]
    star = [([data.uniform(100, 0, 50, 1)], [0]), ([data.permutation(50, 2), data.uniform(50, 0, 9, 3)], [0, 1])]
    chain = data.chain_relations(4000, 600, 4, seed=5)
    if beside != "nothing":
        rels = star if beside == "star" else chain
        queries.insert(1, ("NORMAL", rels, O.mhj(rels)))
    with Context(0) as ctx, ctx.batch() as b:
        for qt, rels, _ in queries:
            b.submit(qt, [ctx.relation(c, a) for c, a in rels])
        for graph in (False, True, True):
            r = b.run(use_graph=graph)
            assert list(zip(r.counts, r.checksums)) == [w for _, _, w in queries]
