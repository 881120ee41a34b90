"""Programs at the edges of the rules that pick a fixpoint's form (hash sets,
row gathers, resident loops, linear recursion), against the CPU oracle."""
import threading

import numpy as np
import pytest

import programs as P
import workloads as W
from gdlog_b200 import DELTA, FULL, INNER, NEWT, OUTER, PLUS, Engine, GdlError

pytestmark = pytest.mark.gpu


def both(prog, *args, mode=None):
    with Engine("gpu", dedup=mode) as g:
        got = prog(g, *args)
    with Engine("oracle") as o:
        want = prog(o, *args)
    assert got == want
    return got


def state(lie, *rels):
    return [(r.size(), r.digest()) for r in rels] + [lie.trace().tolist()]


def tmp_joined_into_itself(eng, edges, sel):
    """tmp :- edge, tmp: the join reads the NEWT that it appends to, as it was
    when the join began."""
    edge = eng.relation("edge")
    out = eng.relation("out", index_flag=False)
    tmp = eng.relation("tmp", index_flag=False, tmp_flag=True)
    eng.load(edge, edges)
    eng.load(out, edges[::3])
    eng.load(tmp, None)
    lie = eng.lie()
    lie.add_relations(edge, True)
    lie.add_relations(out, False)
    lie.add_tmp_relation(tmp)
    lie.add_join(edge, FULL, out, DELTA, tmp, (OUTER(1), INNER(1)))
    lie.add_join(edge, FULL, tmp, NEWT, tmp, sel)
    lie.add_join(edge, FULL, tmp, NEWT, out, (OUTER(1), INNER(1)))
    return [lie.fixpoint()] + state(lie, out)


@pytest.mark.parametrize("sel", [(OUTER(1), INNER(1)), (INNER(1), OUTER(1))])
@pytest.mark.parametrize("base,mode", [(0, None), (0, "dense_rows"), (70000, None),
                                       (70000, "sort")])
def test_tmp_joined_into_itself(base, mode, sel):
    """Ids below 2^13 (bitmaps) and from 70,000 on (lists)."""
    edges = W.rmat_edges(13, 3000, seed=8) + np.uint64(base)
    got = both(tmp_joined_into_itself, edges, sel, mode=mode)
    assert got[0] > 2


def many_path_relations(eng, n, edges, first):
    """n relations with a dependent column in one LIE; the last is derived."""
    edge = eng.relation("edge")
    paths = [eng.relation(f"path{i}", arity=3, dependent_column_size=1, index_flag=False)
             for i in range(n)]
    for i, p in enumerate(paths):
        eng.load(p, first[i % 3::3])
    eng.load(edge, W.reverse(edges))
    lie = eng.lie()
    lie.add_relations(edge, True)
    for p in paths:
        lie.add_relations(p, False)
    last = paths[-1]
    lie.add_join(edge, FULL, last, DELTA, last, (INNER(1), OUTER(1), PLUS(OUTER(2), 1)))
    return [lie.fixpoint()] + state(lie, *paths)


@pytest.mark.parametrize("n", [31, 33, 40])
def test_asides_of_many_relations(n):
    """Tuples that differ in a dependent column only are put aside until the
    joins are done, whatever the relation's place in the LIE."""
    rng = np.random.default_rng(n)
    edges = W.layered_dag(7, 9, 3)
    first = np.stack([rng.integers(0, 63, 600), rng.integers(0, 8, 600),
                      rng.integers(1, 6, 600)], axis=1).astype(np.uint64)
    got = []
    for mode in (None, "sort"):
        with Engine("gpu", dedup=mode) as g:
            got.append(many_path_relations(g, n, edges, first))
    assert got[0] == got[1]
    assert got[0][n][0] > 2 * 200  # (the derived relation grew)


def hidden_delta(eng, ids, order):
    """Operators around one whose inner is empty, which zeroes its outer's
    DELTA for the operators after it in the LIE and for no others."""
    rng = np.random.default_rng(ids)
    rel = {k: eng.relation(k, index_flag=False) for k in "abc"}
    rel["t"] = eng.relation("t", index_flag=False, tmp_flag=True)
    for k in "efz":
        rel[k] = eng.relation(k)
    for k, n in dict(a=ids // 4, b=ids // 8, c=ids // 8, e=ids, f=ids).items():
        rows = rng.integers(0, ids, size=(n, 2))
        rows[0] = ids - 1
        eng.load(rel[k], rows.astype(np.uint64))
    for k in "zt":
        eng.load(rel[k], None)
    lie = eng.lie()
    for k in "efz":
        lie.add_relations(rel[k], True)
    for k in "abc":
        lie.add_relations(rel[k], False)
    lie.add_tmp_relation(rel["t"])
    for rule in order.split():
        out, outer, inner = rule
        lie.add_join(rel[inner], FULL, rel[outer], NEWT if outer == "t" else DELTA, rel[out],
                     (OUTER(1), INNER(1)))
    lie.max_iteration = 6
    return [lie.fixpoint()] + state(lie, rel["a"], rel["b"], rel["c"])


@pytest.mark.parametrize("ids", [300, 700, 1500, 3000])
@pytest.mark.parametrize("order", [
    "tae bte taf cte caz abe",   # the empty inner last, of a step without a conflict
    "tae bte taz caf abe",       # ... in the middle, an operator without a conflict after it
    "caz tae bte abe",           # ... first
    "tae btz cte caf abe",       # a tmp outer emptied before its second reader
])
def test_empty_inner_hides_a_delta_in_operator_order(ids, order):
    both(hidden_delta, ids, order)
    both(hidden_delta, ids, order, mode="dense_push")


@pytest.mark.parametrize("quirks", ["pull_quirks", "rows_quirks", "static_outer_quirks"])
def test_quirks_in_the_default_forms(quirks):
    import test_pull
    both(getattr(test_pull, quirks))


def copied_over(eng, ids, again):
    """A column-swapping ACopy into a relation whose NEWT a join with a
    transposed output wrote before: the copy replaces that NEWT."""
    rng = np.random.default_rng(ids)
    x, y, a = (eng.relation(k, index_flag=False) for k in "xya")
    e = eng.relation("e")
    for r, n in ((x, 9), (y, ids // 8), (a, ids // 4), (e, ids)):
        rows = rng.integers(0, ids, size=(n, 2))
        rows[0] = ids - 1
        eng.load(r, rows.astype(np.uint64))
    lie = eng.lie()
    lie.add_relations(e, True)
    for r in (x, y, a):
        lie.add_relations(r, False)
    lie.add_join(e, FULL, y, DELTA, y, (OUTER(1), INNER(1)))
    lie.add_join(e, FULL, a, DELTA, x, (INNER(1), OUTER(1)))
    lie.add_acopy(y, x, P.CP_SWAP)
    if again:
        lie.add_join(e, FULL, x, DELTA, x, (INNER(1), OUTER(1)))
        lie.add_join(e, FULL, x, DELTA, a, (OUTER(1), INNER(1)))
    lie.max_iteration = 6
    return [lie.fixpoint()] + state(lie, x, y, a)


@pytest.mark.parametrize("again", [False, True])
@pytest.mark.parametrize("ids", [300, 700, 1500, 3000, 5000])
def test_acopy_replaces_what_a_transposed_output_wrote(ids, again):
    both(copied_over, ids, again)
    both(copied_over, ids, again, mode="dense_push")


def closure_of_a_hidden_relation(eng, edges, shift):
    """A first LIE zeroes edge's count (it is the outer of an empty inner,
    src/join.cu:42-45); the closure over it then derives nothing."""
    edge = eng.relation("edge")
    none = eng.relation("none")
    other = eng.relation("other", index_flag=False)
    path = eng.relation("path", index_flag=False)
    rows = np.concatenate([edges, edges | np.uint64(1 << shift)]) if shift else edges
    eng.load(edge, W.reverse(rows))
    eng.load(path, rows)
    eng.load(none, None)
    eng.load(other, None)
    first = eng.lie()
    first.add_relations(none, True)
    first.add_relations(edge, True)
    first.add_relations(other, False)
    first.add_join(none, FULL, edge, FULL, other, (OUTER(1), INNER(1)))
    it0 = first.fixpoint()
    lie = eng.lie()
    lie.add_relations(edge, True)
    lie.add_relations(path, False)
    lie.add_join(edge, FULL, path, DELTA, path, P.REORDER_PATH)
    it = [it0, lie.fixpoint()]
    if shift:
        return it + [path.instance_stats(2)[0].tolist()]
    return it + state(lie, path)


def test_closure_over_a_relation_that_counts_as_empty():
    e = W.grid_edges(17, 23)
    got = both(closure_of_a_hidden_relation, e, 0)
    assert got[2][0] == len(e)
    both(closure_of_a_hidden_relation, e, 0, mode="dense_push")


def test_batched_closure_over_a_relation_that_counts_as_empty(monkeypatch):
    e = W.grid_edges(5, 8)
    got = []
    for no_graph in (False, True):
        if no_graph:
            monkeypatch.setenv("GDLOG_NO_GRAPH", "1")
        with Engine("gpu") as g:
            shift = g.set_instances([40, 40])
            got.append(closure_of_a_hidden_relation(g, e, shift))
    assert got[0] == got[1]
    assert got[0][2] == [len(e), len(e)]


@pytest.mark.parametrize("bad,refused", [
    (((1 << 10) | 3, 599), True), (((1 << 10) | 7, 599), True), ((31, (1 << 10) | 7), True),
    ((599, 600), True), ((1 << 10, 599), False), ((0, (1 << 10) | 8), False)])
def test_first_tuples_out_of_their_instance(bad, refused, monkeypatch):
    """A batched closure whose path holds a tuple between instances, or past
    an instance's nodes (the edges do not): what the general path does, which
    refuses the tuples derived from it."""
    def run():
        with Engine("gpu") as g:
            assert g.set_instances([600, 8]) == 10
            small = W.grid_edges(2, 4)
            edges = np.concatenate([W.grid_edges(20, 30), small | np.uint64(1 << 10)])
            edge = g.relation("edge")
            path = g.relation("path", index_flag=False)
            g.load(edge, W.reverse(edges))
            g.load(path, np.concatenate([edges, np.array([bad], dtype=np.uint64)]))
            lie = g.lie()
            lie.add_relations(edge, True)
            lie.add_relations(path, False)
            lie.add_join(edge, FULL, path, DELTA, path, P.REORDER_PATH)
            try:
                lie.fixpoint()
            except GdlError as err:
                return err.code
            sizes, digests = path.instance_stats(2)
            return sizes.tolist(), digests.tolist()

    got = run()
    assert isinstance(got, int) == refused
    monkeypatch.setenv("GDLOG_NO_GRAPH", "1")
    assert got == run()


@pytest.mark.parametrize("polls_log2", [6, 7])
def test_wait_limit_of_a_look_back_is_not_the_barriers(polls_log2):
    """A block waits at a resident loop's barrier for the others' steps (here
    over 100 us, some 200 polls), which a limit that suits a look-back must
    not cut short."""
    args = W.cspa_facts(2000, 4000, 1500, seed=1)
    with Engine("gpu") as g:
        want = P.cspa(g, *args).relations["value_alias"].digest()
        g.clear()
        g.set_tuning(spin_limit_log2=polls_log2)
        assert P.cspa(g, *args).relations["value_alias"].digest() == want


def test_engines_on_threads_take_turns_with_resident_loops():
    """Engines of several threads, one of them dropped and made again between
    its queries: resident loops run one at a time, each query's answer is its
    own."""
    queries = [(P.tc, (W.grid_edges(16, 16),)), (P.sg, (W.rmat_edges(10, 4096, seed=1),)),
               (P.cspa, W.cspa_facts(150, 300, 100, seed=1)),
               (P.tc, (W.layered_dag(5, 301, 2) + np.uint64(1 << 20),))]

    def answers(eng, k):
        prog, args = queries[k % len(queries)]
        eng.clear()
        return [(r.size(), r.digest()) for r in prog(eng, *args).relations.values()]

    with Engine("gpu") as g:
        want = [answers(g, k) for k in range(len(queries))]
    wrong = []

    def work(t):
        try:
            eng = Engine("gpu")
            for k in range(40):
                if t == 0 and k % 5 == 4:
                    eng.close()
                    eng = Engine("gpu")
                if answers(eng, t + k) != want[(t + k) % len(queries)]:
                    wrong.append((t, k))
            eng.close()
        except Exception as exc:
            wrong.append((t, repr(exc)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert wrong == []


@pytest.mark.parametrize("scale,edges", [(8, 900), (10, 3000), (11, 7000)])
def test_paths_derived_again_with_other_lengths(scale, edges):
    """Most candidates of a random graph meet their pair in FULL, shorter:
    the lengths are a breadth-first search's."""
    e = W.rmat_edges(scale, edges, seed=scale)
    adj = np.zeros((1 << scale, 1 << scale), dtype=np.float32)
    adj[e[:, 0].astype(int), e[:, 1].astype(int)] = 1
    want, new, length = np.zeros(adj.shape, dtype=np.uint64), adj > 0, 1
    while new.any():
        want[new] = length
        new = (adj @ new.astype(np.float32) > 0) & (want == 0)
        length += 1
    pairs = np.argwhere(want)
    want = np.concatenate([pairs.astype(np.uint64), want[want > 0][:, None]], axis=1)
    for mode in (None, "sort"):
        with Engine("gpu", dedup=mode) as g:
            r = P.path_length(g, e)
            assert r.iterations["plen"] == length - 1
            assert np.array_equal(r.relations["path"].rows(), want)


@pytest.mark.parametrize("ids", [8449, 16384, 20000])
def test_closure_with_a_hub(ids):
    """More sources of one node than linear recursion's form takes: rows
    gathered along in-edges, an update pass with nothing transposed, over
    sides of 34, 64 and 79 tiles."""
    rng = np.random.default_rng(ids)
    e = np.concatenate([rng.integers(0, ids, (ids // 2, 2)),
                        np.stack([np.arange(99), np.full(99, ids - 1)], axis=1)]).astype(np.uint64)
    got = []
    for mode in (None, "dense_push"):
        with Engine("gpu", dedup=mode) as g:
            r = P.tc(g, e)
            got.append([r.iterations] + state(r.lies["tc"], r.output))
    assert got[0] == got[1]


@pytest.mark.parametrize("n", [(1 << 18) + 1, (1 << 19) + 77])
@pytest.mark.parametrize("arity", [2, 3])
def test_second_export_in_pieces(n, arity):
    """A first export below 2^22 rows comes over in one copy, a second one of
    the size in pieces: the same rows."""
    rng = np.random.default_rng(n)
    rows = np.stack([rng.integers(0, 4000, n + 5000), rng.integers(0, 4096, n + 5000)] +
                    [rng.integers(0, 1000, n + 5000)] * (arity == 3), axis=1).astype(np.uint64)
    want = np.unique(rows, axis=0)[:n]
    with Engine("gpu") as g:
        r = g.relation("r", arity=arity)
        g.load(r, want[rng.permutation(len(want))])
        for _ in range(3):
            assert np.array_equal(r.rows(), want)


@pytest.mark.parametrize("n,facts", [(2100, 0.3), (4097, 0.2), (8300, 0.1), (16385, 0.05)])
def test_products_of_sparse_relations(n, facts):
    """Rows around an eighth and a sixteenth of the ids, where listed keys and
    tables meet, at each width of a row."""
    args = W.cspa_facts(n, int(2 * n * facts), int(0.75 * n * facts), seed=2)
    args[0][0] = (n - 1, 0)

    def run(eng):
        r = P.cspa(eng, *args)
        return [r.iterations] + [state(r.lies["analysis"], *r.relations.values())]

    got = []
    for mode in (None, "dense_push"):
        with Engine("gpu", dedup=mode) as g:
            got.append(run(g))
    assert got[0] == got[1]


def test_a_full_beyond_the_list_limit_is_not_read_as_a_list():
    """32,768 sources and 32,767 targets of one node: 2^30 pairs and more, a
    FULL that is kept as a bitmap.  A later LIE that reads it, as an inner or
    as an outer, or derives into it, is refused; the relation stays as it is."""
    k = np.arange(32768)
    edges = np.concatenate([np.stack([k + 1, np.zeros_like(k)], axis=1),
                            np.stack([np.zeros_like(k), k + 32769], axis=1)[:-1]]).astype(np.uint64)
    total = len(edges) + 32768 * 32767
    assert total > (1 << 30) - 4096 and edges.max() < 1 << 16
    with Engine("gpu") as g:
        path = P.tc(g, edges).output
        assert path.size() == total
        out = g.relation("out", index_flag=False)
        other = g.relation("other")
        g.load(out, edges[:5])
        g.load(other, edges[:5])
        digest = path.digest()
        for inner, outer, ver, update in ((path, out, DELTA, out), (other, path, FULL, out),
                                          (other, path, DELTA, path)):
            lie = g.lie()
            lie.add_relations(other, True)
            if update is not path:
                lie.add_relations(path, True)
            lie.add_relations(update, False)
            lie.add_join(inner, FULL, outer, ver, update, (OUTER(1), INNER(1)))
            with pytest.raises(GdlError) as err:
                lie.fixpoint()
            assert err.value.code == 4
            assert (path.size(), path.digest()) == (total, digest)


def static_join_and_copy(eng, ids, base, kind):
    """A join of two static relations whose output's NEWT an ACopy replaces,
    or a Copy from an empty source empties in the first iteration only: its
    tuples are not in FULL after the iteration that ran it."""
    rng = np.random.default_rng(ids)
    s, f, none = eng.relation("s"), eng.relation("f"), eng.relation("none")
    u, v = eng.relation("u", index_flag=False), eng.relation("v", index_flag=False)
    for r, n in ((s, ids // 2), (f, ids // 2), (u, ids // 8), (v, ids // 8)):
        eng.load(r, rng.integers(0, ids, size=(n, 2)).astype(np.uint64) + np.uint64(base))
    eng.load(none, None)
    lie = eng.lie()
    for r in (s, f, none):
        lie.add_relations(r, True)
    for r in (u, v):
        lie.add_relations(r, False)
    lie.add_join(s, FULL, f, FULL, u, (OUTER(1), INNER(1)))
    lie.add_join(s, FULL, v, DELTA, v, (OUTER(1), INNER(1)))
    if kind == "copy":
        lie.add_copy(none, FULL, u, P.CP_SWAP)
    else:
        lie.add_acopy(v, u, P.CP_SWAP if kind == "swap" else (0, 1))
    lie.max_iteration = 6
    return [lie.fixpoint()] + state(lie, u, v)


@pytest.mark.parametrize("kind", ["copy", "swap", "acopy"])
@pytest.mark.parametrize("ids,base", [(200, 0), (1500, 0), (5000, 0), (300, 1 << 20)])
def test_static_join_before_a_copy(ids, base, kind):
    both(static_join_and_copy, ids, base, kind)
    both(static_join_and_copy, ids, base, kind, mode="dense_push")
