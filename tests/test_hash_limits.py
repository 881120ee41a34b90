"""The hash form (csrc/hash.cuh) where its sets and lists run out: iterations
that pass the first set by millions of tuples, and probe chains that no larger
set shortens.  Contents, loop passes and traces are whole numbers and equal the
sorted lists'."""
import os
import subprocess
import sys

import numpy as np
import pytest

import programs as P
import workloads as W
from gdlog_b200 import DELTA, FULL, INNER, OUTER, PLUS, Engine

pytestmark = pytest.mark.gpu

BASE = 1 << 20  # ids beyond the bitmaps


def layered(layers, width, degree, seed):
    """Every node has `degree` sources in the layer before its own; edges in
    the order of the layers."""
    rng = np.random.default_rng(seed)
    dst = np.repeat(np.arange(width, layers * width), degree)
    src = (dst // width - 1) * width + rng.integers(0, width, len(dst))
    return np.unique(np.stack([src, dst], axis=1), axis=0).astype(np.uint64) + np.uint64(BASE)


def outcome(prog, args, mode=None):
    with Engine("gpu", dedup=mode) as g:
        r = prog(g, *args)
        return ({k: (v.size(), v.digest()) for k, v in r.relations.items()}, r.iterations,
                {k: lie.trace().tolist() for k, lie in r.lies.items()})


@pytest.mark.parametrize("degree,width", [(8, 125000), (30, 9000), (100, 3200)])
@pytest.mark.parametrize("prog", ["tc", "path_length"])
def test_first_iteration_passes_the_first_set(prog, degree, width):
    """The first set holds 6.3 million tuples; the first iteration derives
    more than that, nearly all of them new, from runs of `degree` tuples."""
    edges = layered(3, width, degree, degree)
    got = outcome(getattr(P, prog), (edges,))
    assert max(size for size, _ in got[0].values()) - len(edges) > 6_000_000
    assert got == outcome(getattr(P, prog), (edges,), "sort")


def lengths_of_one_pair(eng, n):
    """path(b, y, l + 1) :- edge(a, b), path(a, y, l) from n lengths of one
    pair: every iteration derives n tuples of one prefix."""
    edge = eng.relation("edge")
    path = eng.relation("path", arity=3, dependent_column_size=1, index_flag=False)
    first = np.stack([np.full(n, 3), np.full(n, 60), 2 * np.arange(n)], axis=1)
    eng.load(path, first.astype(np.uint64))
    eng.load(edge, np.array([[3, 4], [4, 5], [4, 6], [6, 7]], dtype=np.uint64))
    lie = eng.lie()
    lie.add_relations(edge, True)
    lie.add_relations(path, False)
    lie.add_join(edge, FULL, path, DELTA, path, (INNER(1), OUTER(1), PLUS(OUTER(2), 1)))
    it = lie.fixpoint()
    return it, path.size(), path.digest(), lie.trace().tolist()


@pytest.mark.parametrize("n", [2047, 2049, 5000])
def test_many_tuples_of_one_prefix_in_one_iteration(n):
    got = []
    for mode in (None, "sort"):
        with Engine("gpu", dedup=mode) as g:
            got.append(lengths_of_one_pair(g, n))
    assert got[0] == got[1]
    assert got[0][1] == 5 * n  # (four nodes are reached from the pair's first)


@pytest.mark.parametrize("n", [2048, 2049, 200000])
def test_many_rows_of_one_prefix_loaded(n):
    """FULL's rows of one pair share a probe chain when the set is filled."""
    got = []
    for mode in (None, "sort"):
        with Engine("gpu", dedup=mode) as g:
            got.append(lengths_of_one_pair(g, n))
    assert got[0] == got[1]
    assert got[0][1] == 5 * n


def test_form_left_in_one_program_is_taken_in_the_next():
    """A loop that went on on sorted lists leaves nothing behind."""
    e = W.grid_edges(20, 20)
    with Engine("gpu") as g:
        want = P.path_length(g, e).relations["path"].digest()
        g.clear()
        lengths_of_one_pair(g, 5000)
        g.clear()
        assert P.path_length(g, e).relations["path"].digest() == want
        g.clear()
        assert P.tc(g, e).output.size() == W.grid_tc_size(20, 20)


def test_pieces_past_the_record_buffer():
    """2.2 million outer rows meet a run of 6,145 tuples, four pieces each:
    more than the record buffer holds.  The run's reservation that straddles
    the buffer's end is expanded by its own warp, like those past it."""
    n, run, hub = 2_200_002, 6145, 5
    rows = np.stack([np.full(n, hub), np.arange(n) + 100000], axis=1).astype(np.uint64)
    run_rows = np.stack([np.full(run, hub), 3_000_000 + 2 * np.arange(run)],
                        axis=1).astype(np.uint64)
    with Engine("gpu") as g:
        edge = g.relation("edge")
        out = g.relation("out", index_flag=False)
        g.load(out, rows)
        g.load(edge, run_rows)
        lie = g.lie()
        lie.add_relations(edge, True)
        lie.add_relations(out, False)
        lie.add_join(edge, FULL, out, DELTA, out, (INNER(1), INNER(0)))
        assert lie.fixpoint() == 2
        got = out.rows()
    assert np.array_equal(got, np.concatenate([rows, run_rows[:, ::-1]]))


MEMORY = """
import sys
sys.path[:0] = sys.argv[1:3]
import torch
import test_hash_limits as T
torch.zeros(1, device="cuda")
before = torch.cuda.mem_get_info()[0]
with T.Engine("gpu") as g:
    T.twenty_relations(g)
    torch.cuda.synchronize()
    print((before - torch.cuda.mem_get_info()[0]) >> 20)
"""


def twenty_relations(eng):
    edge = eng.relation("edge")
    paths = [eng.relation(f"p{i}", arity=3, dependent_column_size=1, index_flag=False)
             for i in range(20)]
    for p in paths:
        eng.load(p, np.array([[1, 2, 3]], dtype=np.uint64))
    eng.load(edge, np.array([[1, 0]], dtype=np.uint64))
    lie = eng.lie()
    lie.add_relations(edge, True)
    for p in paths:
        lie.add_relations(p, False)
    for p in paths[:10]:
        lie.add_join(edge, FULL, p, DELTA, p, (INNER(1), OUTER(1), PLUS(OUTER(2), 1)))
    assert lie.fixpoint() == 2
    assert [p.size() for p in paths] == [2] * 10 + [1] * 10


def test_small_programs_take_little_memory():
    """Twenty relations of one tuple: the lists and sets follow the input (in
    a process of its own, whose memory pool starts empty)."""
    here = os.path.dirname(os.path.abspath(__file__))
    pkg = os.path.join(os.path.dirname(here), "gdlog-multinode_b200")
    out = subprocess.run([sys.executable, "-c", MEMORY, here, pkg], stdout=subprocess.PIPE,
                         text=True, timeout=300, check=True).stdout
    assert int(out) < 256


@pytest.mark.parametrize("prog", ["tc", "path_length"])
def test_a_first_set_sized_for_its_input_grows(prog):
    """4,400 edges through one node derive 4.84 million pairs at once, more
    than the 1,024 for an edge that the first set has room for."""
    k = np.arange(2200)
    edges = np.concatenate([np.stack([k, np.full(2200, 5000)], axis=1),
                            np.stack([np.full(2200, 5000), k + 6000], axis=1)])
    args = (edges.astype(np.uint64) + np.uint64(BASE),)
    got = outcome(getattr(P, prog), args)
    assert got[0]["path"][0] == 4400 + 2200 * 2200
    assert got == outcome(getattr(P, prog), args, "sort")
