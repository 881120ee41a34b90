"""The forms a fixpoint takes by domain, program and size, each against the
general path on the same input: relation contents, loop passes and traces are
whole numbers and equal.

* boolean products (csrc/product.cuh) and the resident loop (csrc/loop.cuh)
  against pushed joins, around the sizes where tiles, words and kernels change;
* linear recursion (csrc/closure.cuh) against pushed joins and, batched,
  against each instance alone: in-degrees at the bound and past it, one-node
  and empty inputs, edges out of the instances;
* hash sets (csrc/hash.cuh) against sorted lists: ids up to the largest, long
  runs, predicates, growth, and dependent columns whose tuples of one
  iteration differ in them alone;
* row export in pieces (gdl_relation_export) around a piece's size.
"""
import os

import numpy as np
import pytest

import batch as B
import programs as P
import workloads as W
from gdlog_b200 import DELTA, FULL, INNER, NEWT, OUTER, PLUS, PRED_LT, Engine, GdlError

pytestmark = pytest.mark.gpu


def outcome(prog, args, mode=None, no_graph=False):
    if no_graph:
        os.environ["GDLOG_NO_GRAPH"] = "1"
    try:
        with Engine("gpu", dedup=mode) as g:
            r = prog(g, *args)
            return ({k: (v.size(), v.digest()) for k, v in r.relations.items()}, r.iterations,
                    {k: lie.trace().tolist() for k, lie in r.lies.items()})
    finally:
        os.environ.pop("GDLOG_NO_GRAPH", None)


@pytest.mark.parametrize("n", [40, 130, 256, 257, 520, 700, 1030, 2050, 4100])
def test_products_equal_pushed_joins(n):
    args = W.cspa_facts(n, 2 * n, 3 * n // 4, seed=n)
    want = outcome(P.cspa, args, "dense_push")
    assert outcome(P.cspa, args) == want
    assert outcome(P.cspa, args, no_graph=True) == want


@pytest.mark.parametrize("nodes,edges", [(200, 300), (256, 900), (700, 1500), (1500, 4000),
                                         (3000, 6000), (5000, 9000), (8192, 12000)])
def test_resident_loop_equals_pushed_joins(nodes, edges):
    rng = np.random.default_rng(nodes)
    e = np.unique(rng.integers(0, nodes, (edges, 2)) ** 2 // nodes, axis=0).astype(np.uint64)
    want = outcome(P.sg, (e,), "dense_push")
    assert outcome(P.sg, (e,)) == want
    assert outcome(P.sg, (e,), no_graph=True) == want


def star(degree):
    """`degree` sources of one node, and a chain through it."""
    s = np.stack([np.arange(degree) + 10, np.full(degree, 3)], axis=1)
    return np.concatenate([s, [[3, 4], [4, 5], [5, 6]]]).astype(np.uint64)


CLOSURES = {
    "empty": np.zeros((0, 2), dtype=np.uint64),
    "loop": np.array([[7, 7]], dtype=np.uint64),
    "cycle": np.stack([np.arange(300), (np.arange(300) + 1) % 300], axis=1).astype(np.uint64),
    "grid": W.grid_edges(17, 23),
    "dag": W.layered_dag(33, 37, 5),
    "wide_dag": W.layered_dag(9, 3001, 6),
    "degree_64": star(64)[:, ::-1].copy(),
    "degree_65": star(65)[:, ::-1].copy(),
    "fan_in": star(2000),
    "rmat": W.rmat_edges(11, 5000, seed=4),
}


@pytest.mark.parametrize("name", CLOSURES)
def test_closure_equals_pushed_joins(name):
    want = outcome(P.tc, (CLOSURES[name],), "dense_push")
    assert outcome(P.tc, (CLOSURES[name],)) == want


def test_batched_closure_equals_each_alone():
    cases = [CLOSURES[k] for k in ("loop", "grid", "dag", "degree_64")] + \
        [np.array([[0, 1]], dtype=np.uint64), W.grid_edges(1, 31), W.grid_edges(1, 33),
         W.layered_dag(4, 256, 9), W.layered_dag(128, 16, 9), W.grid_edges(2, 128)]
    inst = [(e,) for e in cases]
    with Engine("gpu") as g:
        got = B.run_batched(g, P.tc, inst).results
        alone = B.run_plain_loop(g, P.tc, inst).results
        # one in-degree past the bound: the general path, for all of them
        more = inst + [(CLOSURES["degree_65"],)]
        got2 = B.run_batched(g, P.tc, more).results
        alone2 = B.run_plain_loop(g, P.tc, more).results
    assert got == alone
    assert got2 == alone2


@pytest.mark.parametrize("bad", [(0, 1 << 10), ((1 << 10) | 3, 2), (0, 9), (0, 700), (1023, 3)])
def test_edges_out_of_their_instance(bad, monkeypatch):
    """An edge between instances, or past an instance's nodes: the same tuples
    or the same refusal as on the general path."""
    e = W.grid_edges(2, 4)

    def run():
        with Engine("gpu") as g:
            s = g.set_instances([8, 600])
            assert s == 10
            edges = np.concatenate([e, e | np.uint64(1 << s), np.array([bad], dtype=np.uint64)])
            try:
                r = P.tc(g, edges)
            except GdlError as err:
                return err.code
            sizes, digests = r.output.instance_stats(2)
            return sizes.tolist(), digests.tolist()

    got = run()
    monkeypatch.setenv("GDLOG_NO_GRAPH", "1")
    assert got == run()


def at_ids(e, base):
    return e + np.uint64(base)


WIDE = {
    "dag": (P.tc, (at_ids(W.layered_dag(9, 203, 2), 1 << 20),)),
    "largest_id": (P.tc, (np.array([[2**32 - 1, 2**32 - 1], [5, 2**32 - 1], [2**32 - 1, 7]],
                                   dtype=np.uint64),)),
    "one_past_bitmaps": (P.tc, (np.array([[65535, 65536], [65536, 1], [1, 2]], dtype=np.uint64),)),
    "empty": (P.tc, (np.array([[70000, 70001]], dtype=np.uint64),)),
    "fan_out": (P.tc, (at_ids(star(6000)[:, ::-1].copy(), 100000),)),
    "fan_in": (P.tc, (at_ids(star(6000), 100000),)),
    "sg_dag": (P.sg, (at_ids(W.layered_dag(5, 301, 2), 1 << 24),)),
    "sg_rmat": (P.sg, (at_ids(W.rmat_edges(9, 1500, seed=2), 70000),)),
    "sg_grows": (P.sg, (W.layered_dag(6, 11003, 3),)),
}


@pytest.mark.parametrize("name", WIDE)
def test_hash_sets_equal_sorted_lists(name):
    prog, args = WIDE[name]
    want = outcome(prog, args, "sort")
    assert outcome(prog, args) == want
    assert outcome(prog, args, "dense") == want  # (too wide for bitmaps: sets as well)
    assert outcome(prog, args, no_graph=True) == want


def path_rows(eng, edges, rows, reload=True, most=None):
    """path(a, y, l + 1) :- edge(a, x), path(x, y, l) over given first paths."""
    edge = eng.relation("edge")
    path = eng.relation("path", arity=3, dependent_column_size=1, index_flag=False)
    eng.load(path, rows)
    eng.load(edge, W.reverse(edges))
    lie = eng.lie()
    lie.set_reload_full(reload)
    if most is not None:
        lie.max_iteration = most
    lie.add_relations(edge, True)
    lie.add_relations(path, False)
    lie.add_join(edge, FULL, path, DELTA, path, (INNER(1), OUTER(1), PLUS(OUTER(2), 1)))
    it = lie.fixpoint()
    return it, path.rows().tolist(), path.rows(DELTA).tolist(), lie.trace().tolist()


@pytest.mark.parametrize("most", [None, 0, 2])
def test_dependent_columns_that_differ_in_one_iteration(most):
    """First paths of several lengths for one pair, and for pairs that meet in
    one successor: an iteration derives the same (c0, c1) with different
    lengths at once, and all of them are new; a later length is not."""
    rng = np.random.default_rng(1)
    edges = W.layered_dag(7, 9, 3)
    first = np.stack([rng.integers(0, 63, 300), rng.integers(0, 8, 300),
                      rng.integers(1, 6, 300)], axis=1).astype(np.uint64)
    got = []
    for mode in (None, "sort"):
        with Engine("gpu", dedup=mode) as g:
            got.append(path_rows(g, edges, first, most=most))
    assert got[0] == got[1]


def test_hash_predicate_and_tmp():
    """A predicate on generated tuples and a tmp relation between two joins."""
    e = at_ids(W.rmat_edges(8, 900, seed=6), 66000)

    def prog(eng, edges):
        edge = eng.relation("edge")
        out = eng.relation("out", index_flag=False)
        tmp = eng.relation("tmp", index_flag=False)
        eng.load(edge, edges)
        eng.load(out, edges[:50])
        eng.load(tmp, None)
        lie = eng.lie()
        lie.add_relations(edge, True)
        lie.add_relations(out, False)
        lie.add_tmp_relation(tmp)
        lie.add_join(edge, FULL, out, DELTA, tmp, (OUTER(1), INNER(1)))
        lie.add_join(edge, FULL, tmp, NEWT, out, (OUTER(1), INNER(1)), pred=(PRED_LT, 0, 1))
        lie.add_join(edge, FULL, edge, FULL, out, (INNER(1), OUTER(1)), pred=(PRED_LT, 0, 1))
        r = P.Result()
        r.iterations["out"] = lie.fixpoint()
        r.relations["out"], r.lies["out"] = out, lie
        return r

    assert outcome(prog, (e,)) == outcome(prog, (e,), "sort")


@pytest.mark.parametrize("n", [1 << 18, (1 << 18) + 1, (1 << 19) + 77])
@pytest.mark.parametrize("arity", [2, 3])
def test_export_in_pieces(n, arity):
    rng = np.random.default_rng(n)
    rows = np.stack([rng.integers(0, 4000, n + 5000), rng.integers(0, 4096, n + 5000)] +
                    [rng.integers(0, 1000, n + 5000)] * (arity == 3), axis=1).astype(np.uint64)
    want = np.unique(rows, axis=0)[:n]
    with Engine("gpu") as g:
        r = g.relation("r", arity=arity)
        g.load(r, want[rng.permutation(len(want))])
        assert np.array_equal(r.rows(), want)
        with pytest.raises(GdlError):
            import ctypes as C
            out = C.c_uint64(0)
            buf = np.zeros((len(want) - 1, arity), dtype=np.uint64)
            g._call("relation_export", r.id, FULL, buf.ctypes.data_as(C.POINTER(C.c_uint64)),
                    len(want) - 1, C.byref(out))
