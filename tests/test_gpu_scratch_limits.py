"""Calls on a device that is nearly full: what an operator can do without (heads
and filters of bucket indexes, matrices, lists and caches that only save time)
is left out when there is no room for it, and the call gives the same result.

Each test measures the device memory of a call, fills the device up to less than
that but more than the call needs without its optional part, and calls again."""
import contextlib

import numpy as np
import pytest

from accmultiwayjoins_b200 import Context, data
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MB = 1 << 20


def pool_call(name, *args):
    from cuda.bindings import runtime as rt
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert int(err) == 0
    err, *out = getattr(rt, name)(pool, *[getattr(rt.cudaMemPoolAttr, a) if isinstance(a, str) else a for a in args])
    assert int(err) == 0
    return int(out[0]) if out else None


def scratch_of(call):
    """Bytes of device memory that `call` takes on top of what is in use, and its result."""
    import torch
    from cuda.bindings import driver
    torch.cuda.synchronize()
    pool_call("cudaMemPoolTrimTo", 0)
    used = pool_call("cudaMemPoolGetAttribute", "cudaMemPoolAttrUsedMemCurrent")
    pool_call("cudaMemPoolSetAttribute", "cudaMemPoolAttrUsedMemHigh", driver.cuuint64_t(0))
    out = call()
    torch.cuda.synchronize()
    return pool_call("cudaMemPoolGetAttribute", "cudaMemPoolAttrUsedMemHigh") - used, out


@contextlib.contextmanager
def device_with(free, trim=True):
    """The device filled up to `free` bytes (and the pool's unused blocks, unless they are given back first)."""
    import torch
    torch.cuda.synchronize()
    if trim:
        pool_call("cudaMemPoolTrimTo", 0)
    torch.cuda.empty_cache()
    left = torch.cuda.mem_get_info()[0]
    assert left > free
    fill = torch.empty(left - free, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del fill
        torch.cuda.empty_cache()


def path_and_triangles(n, seed):
    """n - 1 edges of a long path (two lists of one candidate each) behind a small graph of triangles."""
    s, d = data.rmat(10, 8000, 0.57, 0.19, 0.19, seed)
    p = np.arange(1024, 1024 + n - len(s), dtype=np.int32)
    return np.concatenate([s, p]), np.concatenate([d, p + 1])


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("share", [0.3, 0.6])   # the pool rounds each block up: some 40 MB
def test_batch_triangles_without_room_for_heads(graph, share):
    s, d = path_and_triangles(1 << 23, 1)
    want = O.triangle(s[:20000], d[:20000])
    heads = 36 << 23
    with Context(0) as ctx:
        e = ctx.relation([s, d], [0, 1])

        def call():
            with ctx.batch() as b:
                b.submit("TRI", [e])
                r = b.run(use_graph=graph)
                return r.counts[0], r.checksums[0]
        need, got = scratch_of(call)
        assert got == want and need > heads
        with device_with(need - int(share * heads)):
            assert call() == want
        assert call() == want


@pytest.mark.parametrize("kind", ["hub_source", "bag", "sparse"])
@pytest.mark.parametrize("n", [1, 33, 700, 5000])
def test_batch_triangles_with_and_without_heads(kind, n):
    """A context with a memory budget that the heads do not fit."""
    rng = np.random.default_rng(n)
    if kind == "hub_source":
        s, d = data.rmat(9, n, 0.57, 0.19, 0.19, n)
    elif kind == "bag":
        s, d = rng.integers(-20, 20, (2, n)).astype(np.int32)
    else:
        s, d = (rng.integers(0, 60, (2, n)) * 65536 + 7).astype(np.int32)
    want = O.triangle(s, d)
    launches = []
    for budget in (0, 1):
        with Context(0, mem_budget=budget) as ctx, ctx.batch() as b:
            b.submit("TRI", [ctx.relation([s, d], [0, 1])])
            b.submit("TRI", [ctx.relation([d, s], [0, 1])])
            for graph in (False, True, True):
                r = b.run(use_graph=graph)
                assert (r.counts[0], r.checksums[0]) == want
                assert (r.counts[1], r.checksums[1]) == O.triangle(d, s)
            launches.append(r.launches)
    assert launches[1] == launches[0] - 1   # the heads' kernel


def test_breadth_first_triangles_without_room_for_the_hub_matrix():
    """A complete graph of 200 vertices with its ids spread over 20 thousand: 1.3
    million candidates over 20 thousand edges, and a matrix of 32 MB."""
    u, v = np.triu_indices(200, 1)
    s, d = (u * 100).astype(np.int32), (v * 100).astype(np.int32)
    want = O.triangle(s, d)
    with Context(0) as ctx:
        e = ctx.relation([s, d], [0, 1])
        assert (lambda r: (r.count, r.checksum))(ctx.lftj([e], algo="BFS")) == want
        pool_call("cudaMemPoolTrimTo", 0)
        assert (lambda r: (r.count, r.checksum))(ctx.lftj([e], algo="DFS")) == want   # the pool's first block
        with device_with(8 * MB, trim=False):
            got = ctx.lftj([e], algo="BFS")
            assert (got.count, got.checksum) == want


def result(r):
    return r.count, r.checksum


def test_chain_counts_without_room_for_heads_and_lists():
    """8M probe rows and small build relations: the lists of what the flat
    kernel leaves (12 bytes a probe row) are nearly all of the query's memory;
    the frontier kernel joins it without them."""
    n = 1 << 23
    rels = [([data.uniform(n, 0, 4000, 1), data.uniform(n, 0, 4000, 2)], [0, 1])]
    rels += [([data.uniform(1000, 0, 4000, 3 + i), data.uniform(1000, 0, 4000, 7 + i)], [1 + i, 2 + i]) for i in range(2)]
    with Context(0) as ctx:
        hs = [ctx.relation(c, at) for c, at in rels]
        want = result(ctx.amhj("NORMAL", hs, plan="frontier"))
        assert want[0] > 0
        need, got = scratch_of(lambda: result(ctx.amhj("NORMAL", hs)))
        assert got == want and need > 12 << 23
        with device_with(need // 2):
            assert result(ctx.amhj("NORMAL", hs)) == want


def test_indexes_built_together_or_one_by_one():
    """A wide small table beside a long narrow one: built together they share
    columns as many and as long as any needs, built one by one they do not."""
    n = 1 << 23
    wide = [data.uniform(100, 0, 1 << 20, 3 + i) for i in range(4)]
    rels = [([data.uniform(1000, 0, 100, 1), data.uniform(1000, 0, n, 2)], [0, 1]),
            ([data.permutation(n, 8), data.uniform(n, 0, 1 << 20, 9)], [1, 2]), (wide, [0, 3, 4, 5])]
    rels[2][0][0][:] = np.arange(100)
    want = O.mhj(rels)
    with Context(0) as ctx:
        hs = [ctx.relation(c, at) for c, at in rels]
        need, got = scratch_of(lambda: result(ctx.amhj("NORMAL", hs)))
        assert got == want and want[0] == 1000 and need > 23 << 23   # 4 columns, bounds, places
        with device_with(need - (5 << 23)):                          # 2 columns fewer: 8 bytes a row
            assert result(ctx.amhj("NORMAL", hs)) == want
