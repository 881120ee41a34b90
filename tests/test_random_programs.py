"""Random programs against the CPU oracle: one or two LIEs of joins, Copies and
swapping ACopies over static, update and tmp relations (some of them empty),
ids below 2^8, 2^11 and 2^13 and beyond the bitmaps.  Every size, digest, DELTA,
loop-pass count and trace is equal."""
import random

import numpy as np
import pytest

from gdlog_b200 import DELTA, FULL, INNER, NEWT, OUTER, PRED_LT, PRED_NE, Engine

pytestmark = pytest.mark.gpu

SELS = [(OUTER(1), INNER(1))] * 4 + [(INNER(1), OUTER(1))] * 4 + \
    [(OUTER(0), INNER(1)), (INNER(1), OUTER(0)), (OUTER(1), OUTER(0))]
PREDS = [None] * 6 + [(PRED_NE, 0, 1), (PRED_LT, 0, 1)]


def lie_rules(r, statics, updates, tmps):
    rules = []
    for _ in range(r.randint(1, 7)):
        kind = r.random()
        if kind < 0.10 and len(updates) > 1:
            rules.append(("acopy", *r.sample(updates, 2), r.choice([(1, 0), (1, 0), (0, 1)])))
            continue
        if kind < 0.16:
            src, dst = r.choice(statics + updates), r.choice(updates)
            if src != dst:
                ver = r.choice([FULL, DELTA]) if src in updates else FULL
                rules.append(("copy", src, ver, dst, r.choice([(1, 0), (0, 1)])))
                continue
        inner = r.choice(statics) if r.random() < 0.65 else r.choice(updates)
        kind = r.random()
        outer, ver = (r.choice(tmps), NEWT) if tmps and kind < 0.3 else \
            (r.choice(updates), DELTA) if kind < 0.88 else (r.choice(statics), FULL)
        out = r.choice(tmps) if tmps and r.random() < 0.35 else r.choice(updates)
        rules.append(("join", inner, outer, ver, out, r.choice(SELS), r.choice(PREDS)))
    return rules, r.choice([4, 1, 2, 3, 5]), r.random() < 0.5


def program(seed):
    r = random.Random(seed)
    ids, base = r.choice([(r.randint(20, 255), 0), (r.randint(256, 2040), 0),
                          (r.randint(2060, 4500), 0), (r.randint(40, 400), 1 << 20)])
    sizes = {f"s{i}": 0 if r.random() < 0.2 else int(ids * r.uniform(0.1, 0.5)) + 1
             for i in range(r.randint(2, 3))}
    sizes |= {f"u{i}": 0 if r.random() < 0.15 else int(ids * r.uniform(0.02, 0.25)) + 1
              for i in range(r.randint(1, 3))}
    sizes |= {f"t{i}": 0 for i in range(r.randint(0, 2))}
    kinds = [[k for k in sizes if k[0] == c] for c in "sut"]
    lies = [lie_rules(r, *kinds) for _ in range(r.choice([1, 1, 2]))]
    rng = np.random.default_rng(seed)
    rows = {}
    for k, n in sizes.items():
        rows[k] = rng.integers(0, ids, (n, 2)).astype(np.uint64) + np.uint64(base)
        rows[k][:1] = base + ids - 1
    return rows, lies


def run(kind, rows, lies):
    out = []
    with Engine(kind) as eng:
        rel = {k: eng.relation(k, index_flag=k[0] == "s", tmp_flag=k[0] == "t") for k in rows}
        for k, x in rows.items():
            eng.load(rel[k], x if len(x) else None)
        for rules, most, reload in lies:
            lie = eng.lie()
            lie.set_reload_full(reload)
            for k in rows:
                if k[0] == "t":
                    lie.add_tmp_relation(rel[k])
                else:
                    lie.add_relations(rel[k], k[0] == "s")
            for what, *x in rules:
                if what == "acopy":
                    lie.add_acopy(rel[x[0]], rel[x[1]], x[2])
                elif what == "copy":
                    lie.add_copy(rel[x[0]], x[1], rel[x[2]], x[3])
                else:
                    inner, outer, ver, to, sel, pred = x
                    lie.add_join(rel[inner], FULL, rel[outer], ver, rel[to], sel, pred=pred)
            lie.max_iteration = most
            out.append((lie.fixpoint(), lie.trace().tolist()))
            out += [(k, rel[k].size(), rel[k].digest(), rel[k].size(DELTA))
                    for k in rows if k[0] == "u"]
    return out


@pytest.mark.parametrize("first", range(0, 120, 20))
def test_random_programs_match_the_oracle(first):
    for seed in range(first, first + 20):
        p = program(seed)
        assert run("gpu", *p) == run("oracle", *p), seed
