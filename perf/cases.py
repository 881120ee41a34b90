"""The work this engine is used for, as cases that can be timed.

A case is one program (transitive closure, same generation, points-to
analysis, path lengths, or a batch of closures) over one input.  A pass is
what a program using the engine does with a query: drop the previous
program, declare and load the relations, run the fixpoint(s), take the
result.  Binary relations come from device memory and their results go to
buffers in device memory that the program keeps (DeviceRows, export_device);
ternary ones and batches use the host arrays their entry points take.  One
engine serves all queries of the process, as a service or a driver loop
keeps one (and another those with ternary relations, whose keys have a
layout of their own).

All results are whole numbers: the sorted tuples and the loop-pass counts.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gdlog-multinode_b200"))

import batch as B  # noqa: E402
import programs as P  # noqa: E402
import workloads as W  # noqa: E402
from gdlog_b200 import FULL, DeviceRows, Engine  # noqa: E402

# Input ranges.  Layered DAGs as in the batched and the serving workload.
DAG_LAYERS, DAG_WIDTH = (8, 128), (16, 256)
# Ids from 2^16 on: the programs run on sorted lists instead of bitmaps.
WIDE_NODES = 1 << 16


def listed():
    return [
        # the smallest closure (2^8 ids, 30 passes): launches and host calls
        {"name": "tc_grid_16", "kind": "tc_grid", "rows": 16, "cols": 16},
        # the benchmark's 64 x 64 grid closure: many short passes
        {"name": "tc_grid_64", "kind": "tc_grid", "rows": 64, "cols": 64},
        # a reachability query of the serving mix, ragged: 8,113 ids
        {"name": "tc_dag_8k", "kind": "tc_dag", "layers": 61, "width": 133},
        # a sparse dependency graph of 80,000 ids, beyond the bitmaps
        {"name": "tc_dag_wide", "kind": "tc_dag", "layers": 8, "width": 10007},
        # the smallest same-generation query of the serving mix
        {"name": "sg_rmat_s10", "kind": "sg_rmat", "scale": 10, "edges": 4096},
        # the headline benchmark
        {"name": "sg_rmat_s14", "kind": "sg_rmat", "scale": 14, "edges": 40000},
        # the largest same-generation benchmark, 2^16 ids
        {"name": "sg_rmat_s16", "kind": "sg_rmat", "scale": 16, "edges": 120000},
        # same generation over 66,000 ids, beyond the bitmaps
        {"name": "sg_dag_wide", "kind": "sg_dag", "layers": 6, "width": 11003},
        # points-to analysis of a small unit (the benchmark's 300 variables)
        {"name": "cspa_300", "kind": "cspa", "variables": 300},
        # ... and of the full configuration
        {"name": "cspa_20000", "kind": "cspa", "variables": 20000},
        # shortest path lengths (arity 3, host rows in and out)
        {"name": "path_length_grid_64", "kind": "path_length", "rows": 64, "cols": 64},
        # many small closures in one batch (host rows in, one result each)
        {"name": "tc_batch_384", "kind": "tc_batch", "instances": 384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tc_grid", "tc_dag", "tc_dag_wide", "sg_rmat", "sg_dag", "cspa",
                       "path_length", "tc_batch"])
    if kind in ("tc_grid", "path_length"):
        return {"kind": kind, "rows": rng.randint(12, 64), "cols": rng.randint(12, 64)}
    if kind == "tc_dag":
        return {"kind": kind, "layers": _log_int(rng, *DAG_LAYERS),
                "width": _log_int(rng, *DAG_WIDTH)}
    if kind == "tc_dag_wide":
        layers = rng.randint(4, 8)
        return {"kind": "tc_dag", "layers": layers,
                "width": WIDE_NODES // layers + rng.randint(1, 4000)}
    if kind == "sg_dag":
        layers = rng.randint(3, 6)
        return {"kind": kind, "layers": layers,
                "width": WIDE_NODES // layers + rng.randint(1, 2000)}
    if kind == "sg_rmat":
        # sparser above 2^14 ids, as the benchmarks are
        scale = rng.randint(10, 16)
        density = rng.uniform(1.2, 4.0) if scale <= 14 else rng.uniform(1.0, 1.8)
        return {"kind": kind, "scale": scale, "edges": int(density * (1 << scale))}
    if kind == "cspa":
        return {"kind": kind, "variables": _log_int(rng, 100, 16000)}
    return {"kind": kind, "instances": _log_int(rng, 16, 384)}


def _grid(rows, cols, seed):
    """The directed grid with one edge in a hundred (at least one) closed."""
    e = W.grid_edges(rows, cols)
    rng = np.random.default_rng(seed)
    closed = rng.choice(len(e), size=max(1, len(e) // 100), replace=False)
    return np.delete(e, closed, axis=0)


def _facts(case, seed):
    """The input relations of a case as host arrays."""
    kind = case["kind"]
    if kind == "tc_grid":
        return (_grid(case["rows"], case["cols"], seed),)
    if kind == "path_length":
        # junctions numbered in no order
        ids = np.random.default_rng(seed).permutation(case["rows"] * case["cols"])
        return (ids.astype(np.uint64)[W.grid_edges(case["rows"], case["cols"]).astype(np.int64)],)
    if kind in ("tc_dag", "sg_dag"):
        return (W.layered_dag(case["layers"], case["width"], seed),)
    if kind == "sg_rmat":
        return (W.rmat_edges(case["scale"], case["edges"], seed=seed),)
    n = case["variables"]
    return W.cspa_facts(n, 2 * n, 3 * n // 4, seed=seed)


PROGRAM = {"tc_grid": P.tc, "tc_dag": P.tc, "sg_rmat": P.sg, "sg_dag": P.sg, "cspa": P.cspa,
           "path_length": P.path_length, "tc_batch": P.tc}
_engines = {}


def _engine(ternary):
    if ternary not in _engines:
        _engines[ternary] = Engine("gpu")
    return _engines[ternary]


def _capacity(case):
    """Rows of each result buffer: upper bounds where the program has one
    below the square of the ids, else well above what its graphs give."""
    kind = case["kind"]
    if kind == "tc_grid":
        return {"path": W.grid_tc_size(case["rows"], case["cols"])}
    if kind == "tc_dag":
        layers, width = case["layers"], case["width"]
        return {"path": sum(min(width, 2 ** k) * width * (layers - k) for k in range(1, layers))}
    if kind == "sg_dag":
        return {"sg": _sg_dag_bound(case["layers"], case["width"])}
    if kind == "sg_rmat":
        n = 1 << case["scale"]
        return {"sg": n * n if case["scale"] <= 14 else int(1.4 * _sg_rmat_share(case) * n * n)}
    n = case["variables"]
    share = (1.0, 1.0, 1.0) if n < 4096 else (0.35, 0.4, 1.0)
    return dict(zip(("value_flow", "memory_alias", "value_alias"),
                    (int(x * n * n) for x in share)))


def _device_rows(rows):
    """Rows and their column-swapped twin in device memory."""
    t = torch.from_numpy(rows.astype(np.int64)).cuda()
    return DeviceRows(t, t.flip(1).contiguous())


def prepare(case, seed):
    state = {"kind": case["kind"], "engine": _engine(case["kind"] == "path_length")}
    if case["kind"] == "tc_batch":
        dags = W.dag_batch(case["instances"], seed=seed, l_range=DAG_LAYERS, w_range=DAG_WIDTH)
        state["inputs"] = [(e,) for _, _, e in dags]
        state["nodes"] = [layers * width for layers, width, _ in dags]
    elif case["kind"] == "path_length":
        state["inputs"] = _facts(case, seed)
    else:
        state["inputs"] = tuple(_device_rows(x) for x in _facts(case, seed))
        state["results"] = {name: torch.zeros((n, 2), dtype=torch.int64, device="cuda")
                            for name, n in _capacity(case).items()}
    return state


def run(state):
    eng = state["engine"]
    if state["kind"] == "tc_batch":
        res = B.run_batched(eng, P.tc, state["inputs"], state["nodes"]).results
        return {"sizes": np.array([r.sizes["path"] for r in res], dtype=np.int64),
                "digests": np.array([int(r.digests["path"], 16) for r in res],
                                    dtype=np.uint64).view(np.int64),
                "passes": np.array([r.iterations["tc"] for r in res], dtype=np.int64)}
    eng.clear()
    r = PROGRAM[state["kind"]](eng, *state["inputs"])
    out = {"passes_" + name: n for name, n in r.iterations.items()}
    for name, rel in r.relations.items():
        if rel.arity == 3:
            out[name] = rel.rows().view(np.int64)
            continue
        buf = state["results"][name]
        out["size_" + name] = eng.export_device(rel, FULL, buf.data_ptr(), len(buf))
        out[name] = buf
    return out


def _dag_closure(layers, width):
    """Expected closure size: a node reaches reach(k) nodes k layers on."""
    total, reach = 0.0, 1.0
    for k in range(1, layers):
        reach = width * -math.expm1(2 * reach * math.log1p(-1.0 / width))
        total += reach * width * (layers - k)
    return total


def _sg_dag_bound(layers, width):
    """A node shares its generation with siblings by either parent and the
    children of its parents' generation; two children a parent."""
    s = total = 0
    for _ in range(1, layers):
        s = 4 * s + 2
        total += min(s, width) * width
    return total


def _sg_rmat_share(case):
    """|sg| over the square of the ids, fitted to measured sizes."""
    return 0.058 * case["edges"] / (1 << case["scale"]) * 0.89 ** (case["scale"] - 14)


def work(case):
    """Each input row read and each result row written once, 16 bytes a row
    of two columns (24 of three); sizes of results that depend on the drawn
    graph are fitted to measured ones.  No arithmetic counts but the joins'
    comparisons, so no operations are given."""
    kind = case["kind"]
    if kind in ("tc_grid", "path_length"):
        r, c = case["rows"], case["cols"]
        edges, out = 2 * r * c - r - c, W.grid_tc_size(r, c)
        return {"bytes": 16 * edges + (24 if kind == "path_length" else 16) * out, "flops": 0}
    if kind == "tc_dag":
        n = case["layers"] * case["width"]
        return {"bytes": 32 * n + 16 * _dag_closure(case["layers"], case["width"]), "flops": 0}
    if kind == "sg_dag":
        layers, width = case["layers"], case["width"]
        return {"bytes": 32 * layers * width + 16 * _sg_dag_bound(layers, width), "flops": 0}
    if kind == "sg_rmat":
        n = 1 << case["scale"]
        return {"bytes": 16 * case["edges"] + 16 * _sg_rmat_share(case) * n * n, "flops": 0}
    if kind == "cspa":
        n = case["variables"]
        return {"bytes": 16 * 2.75 * n + 16 * 1.39 * n * n, "flops": 0}
    # a batch: its edges, and each closure kept on the device, a bit a pair
    edges = bits = 0
    rng = np.random.default_rng(0)
    for _ in range(case["instances"]):
        n = W.log_uniform_int(rng, *DAG_LAYERS) * W.log_uniform_int(rng, *DAG_WIDTH)
        edges += 2 * n
        bits += n * n
    return {"bytes": 16 * edges + bits / 8, "flops": 0}
