"""The tries of a triangle over three relations: those whose rows can be bucketed
are built together, whatever the others need (repeated rows, rows past the
longest block sort, sparse ranges, no rows at all)."""
import ctypes as C

import numpy as np
import pytest

from accmultiwayjoins_b200 import Context, _lib as L, data
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ATTRS = ([0, 1], [1, 2], [0, 2])


def launches(ctx):
    n = C.c_uint64()
    L.check(L.load().amj_ctx_launch_count(ctx.handle, C.byref(n)))
    return int(n.value)


def i32(*cols):
    return [np.ascontiguousarray(c, np.int32) for c in cols]


def unique(cols):
    u = np.unique(np.stack(cols, 1), axis=0)
    return i32(u[:, 0], u[:, 1])


def check(ctx, rels, algo="DFS"):
    want = O.mhj([(unique(c), a) for c, a in zip(rels, ATTRS)])
    got = ctx.lftj([ctx.relation(c, a) for c, a in zip(rels, ATTRS)], algo=algo)
    assert (got.count, got.checksum) == want
    return got


def test_repeated_rows_cost_a_compaction_not_a_second_build():
    rels = [i32(*data.rmat(12, 30000, 0.57, 0.19, 0.19, s)) for s in (1, 2, 3)]
    with Context(0) as ctx:
        check(ctx, rels)
        n = []
        for repeated in (0, 1, 3):
            r = [i32(*(np.concatenate([c, c[:1]]) for c in cols)) if i < repeated else cols
                 for i, cols in enumerate(rels)]
            before = launches(ctx)
            check(ctx, r)
            n.append(launches(ctx) - before)
        # a scan, the compaction and the row pointers of each such relation
        assert n[1] - n[0] <= 4 and n[2] - n[0] <= 12


FORMS = {
    "plain": lambda c, rng: c,
    "one_repeated": lambda c, rng: [np.concatenate([x, x[-1:]]) for x in c],
    "all_repeated": lambda c, rng: [np.tile(x, 3) for x in c],
    "long_row": lambda c, rng: [np.concatenate([c[0], np.full(33000, -7)]),
                                np.concatenate([c[1], rng.permutation(33000)])],
    "repeated_long_row": lambda c, rng: [np.concatenate([c[0], np.full(33000, 5)]),
                                         np.concatenate([c[1], rng.integers(0, 200, 33000)])],
    "block_row": lambda c, rng: [np.concatenate([c[0], np.full(3000, 5)]), np.concatenate([c[1], rng.integers(0, 2500, 3000)])],
    "sparse": lambda c, rng: [np.concatenate([c[0], [-2000000000, 2000000000]]), np.concatenate([c[1], [0, 0]])],
    "empty": lambda c, rng: [c[0][:0], c[1][:0]],
}


@pytest.mark.parametrize("algo", ["DFS", "BFS"])
@pytest.mark.parametrize("others", ["plain", "all_repeated"])
@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("form", list(FORMS))
def test_one_relation_of_another_form(ctx, form, which, others, algo):
    rng = np.random.default_rng(which)
    base = [i32(*data.rmat(8, 2500, 0.57, 0.19, 0.19, s)) for s in (4, 5, 6)]
    rels = []
    for i, c in enumerate(base):
        c = FORMS[form if i == which else others](c, rng)
        p = rng.permutation(len(c[0]))
        rels.append(i32(c[0][p], c[1][p]))
    check(ctx, rels, algo)


@pytest.mark.parametrize("algo", ["DFS", "BFS"])
def test_all_relations_alone(ctx, algo):
    rng = np.random.default_rng(1)
    base = [i32(*data.rmat(8, 2500, 0.57, 0.19, 0.19, s)) for s in (4, 5, 6)]
    check(ctx, [i32(*FORMS["sparse"](c, rng)) for c in base], algo)
    check(ctx, [i32(*FORMS["long_row"](c, rng)) for c in base], algo)
    check(ctx, [i32(*FORMS["empty"](c, rng)) for c in base], algo)
