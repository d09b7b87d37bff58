"""Performance cases: what programs have this engine do, by size and calling pattern.

Each case loads a seeded graph and evaluates a seeded rule set through one of
the public calling patterns:

    each    GpuRulesLib.evaluate_rule, one call per rule (the Scala caller's pattern)
    batch   GpuRulesLib.evaluate_rules_batch, rule texts in, results out (the miner's pattern)
    replay  GpuRulesLib.prepare_batch once, then PreparedBatch.run + counts (a rule set
            scored again and again)
    serve   GpuServer.submit / poll, a burst of requests drained to the last

Graphs have the shapes of this repository's synthetic configurations (uniform,
dense, dense with skewed subjects, DBpedia-like, biomedical with hubs) and of
its wide-domain test graph.  Loading the graph belongs to `prepare`: a program
does it once.  Results are exact counts; the two ratios follow from them.  The
phase times that the engine reports beside the counts are no results and are
not returned.
"""
from __future__ import annotations

import functools
import math
import os
import tempfile

import numpy as np

import masterthesis_gpu_acceleration_b200 as eng
from masterthesis_gpu_acceleration_b200 import miner

FIELDS = ("support", "headSize", "headSupport", "headCoverage", "bodySize", "confidence")
RESULT = np.dtype([("support", "i4"), ("headSize", "i4"), ("headSupport", "i4"), ("headCoverage", "f8"),
                   ("bodySize", "i4"), ("confidence", "f8"), ("supportMs", "f8"), ("confidenceMs", "f8")], align=True)

# Graph shapes: entities, predicates, triples, Zipf exponents of the predicate
# sizes, subjects and objects (0: uniform), and the in-degree of the hubs (two
# on each of five predicates; 0: none).


def _uniform(entities, predicates, triples):
    return dict(entities=entities, predicates=predicates, triples=triples, pred_zipf=0.0, subj_zipf=0.0, obj_zipf=0.0,
                hub=0)


def _skewed(entities, predicates, triples):
    return dict(entities=entities, predicates=predicates, triples=triples, pred_zipf=1.1, subj_zipf=1.5, obj_zipf=1.3,
                hub=0)


def _bio(entities, triples, hub):
    return dict(entities=entities, predicates=50, triples=triples, pred_zipf=0.0, subj_zipf=0.0, obj_zipf=1.2, hub=hub)


def _rules(kind, count, lo, hi, call):
    return dict(kind=kind, rules=count, min_atoms=lo, max_atoms=hi, call=call)


def listed():
    return [
        # the smallest call: one short rule on a small graph, latency only
        dict(name="one rule, small graph", **_uniform(10_000, 20, 100_000), **_rules("chain", 1, 2, 2, "each")),
        # a rule learner scoring its candidates one call at a time
        dict(name="rule by rule", **_skewed(100_000, 600, 206_000), **_rules("chain", 128, 1, 4, "each")),
        # the same on a graph with hubs, rules crossing them: single heavy rules
        dict(name="hub rules one by one", **_bio(30_000, 680_000, 5_000), **_rules("hub", 20, 2, 4, "each")),
        # a handful of rules on a dense graph in one call
        dict(name="dense batch", **_uniform(2_000, 10, 100_000), **_rules("chain", 10, 2, 3, "batch")),
        # long bodies: up to the eight atoms a rule may have
        dict(name="long rules", **_uniform(10_000, 20, 100_000), **_rules("chain", 200, 4, 8, "batch")),
        # confidences of a fixed rule set on a dense graph with skewed subjects
        dict(name="dense skewed replay", entities=2_000, predicates=10, triples=100_000, pred_zipf=0.0, subj_zipf=1.3,
             obj_zipf=0.0, hub=0, **_rules("chain", 10, 2, 3, "replay")),
        # the headline workload, from rule texts to results
        dict(name="10,000 rules in one call", **_skewed(100_000, 600, 206_000),
             **_rules("chain", 10_000, 1, 4, "batch")),
        # the headline workload prepared once and run again
        dict(name="10,000 rules replayed", **_skewed(100_000, 600, 206_000),
             **_rules("chain", 10_000, 1, 4, "replay")),
        # a fixed rule set on a graph with hubs
        dict(name="biomedical replay", **_bio(30_000, 680_000, 5_000), **_rules("biomedical", 50, 2, 5, "replay")),
        # one level of the rule miner: dangling and closing refinements
        dict(name="miner level", **_skewed(100_000, 600, 206_000), **_rules("mined", 5_000, 2, 3, "batch")),
        # a burst of requests to the serving loop, any length
        dict(name="served burst", **_uniform(10_000, 20, 100_000), **_rules("chain", 1_000, 1, 8, "serve")),
        # more distinct head objects than a block's shared memory has bits for
        dict(name="wide object domain", **_uniform(1_200_000, 3, 1_500_000), **_rules("chain", 6, 1, 3, "batch")),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["uniform", "dense", "skewed", "bio", "mined", "wide"])
    if family == "uniform":   # small graphs, any rule length
        n = _log_int(rng, 3_000, 30_000)
        g = _uniform(n, rng.randint(10, 30), n * rng.randint(7, 10))
        lo = rng.randint(1, 4)
        r = _rules("chain", _log_int(rng, 1, 2_000), lo, rng.randint(lo, 8), rng.choice(["each", "batch", "serve"]))
        if r["call"] == "each":
            r["rules"] = min(r["rules"], 100)
    elif family == "dense":
        n = rng.randint(1_000, 2_000)
        g = _uniform(n, 10, n * rng.randint(30, 50))
        g["subj_zipf"] = rng.choice([0.0, 1.3])
        r = _rules("chain", rng.randint(3, 40), 2, 3, rng.choice(["batch", "replay"]))
    elif family == "skewed":   # DBpedia-like, a few rules to the whole set
        n = _log_int(rng, 20_000, 100_000)
        g = _skewed(n, rng.randint(300, 600), int(n * rng.uniform(1.7, 2.06)))
        r = _rules("chain", _log_int(rng, 30, 9_000), 1, rng.randint(2, 4), rng.choice(["batch", "replay", "each"]))
        if r["call"] == "each":
            r["rules"] = min(r["rules"], 200)
    elif family == "bio":
        n = _log_int(rng, 8_000, 25_000)
        g = _bio(n, n * rng.randint(17, 22), n // 6)
        r = _rules("biomedical", rng.randint(10, 50), 2, rng.randint(3, 5), rng.choice(["each", "replay"]))
        if r["call"] == "each":
            r.update(rules=min(r["rules"], 12), max_atoms=min(r["max_atoms"], 4))
    elif family == "mined":
        n = _log_int(rng, 20_000, 100_000)
        g = _skewed(n, rng.randint(300, 600), int(n * rng.uniform(1.7, 2.06)))
        r = _rules("mined", _log_int(rng, 200, 5_000), rng.randint(1, 2), 3, "batch")
    else:
        n = rng.randint(1_000_000, 1_190_000)
        g = _uniform(n, rng.randint(2, 3), int(n * 1.25))
        r = _rules("chain", rng.randint(1, 6), 1, rng.randint(1, 3), rng.choice(["batch", "each"]))
    return dict(**g, **r)


# ---------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=4)
def _zipf(n, s):
    return np.cumsum(np.arange(1, n + 1, dtype=np.float64) ** -s)


def _zipf_ranks(rng, n, s, count):
    if s <= 0:
        return rng.integers(0, n, count)
    cum = _zipf(n, s)
    return np.minimum(np.searchsorted(cum, rng.random(count) * cum[-1]), n - 1)


def _relabel(rng, n, s):
    """Ranks to entities: its own order for every predicate (ranks of a skewed column)."""
    if s <= 0:
        return lambda k: k
    a = int(rng.integers(1, n))
    while math.gcd(a, n) != 1:
        a = a % n + 1
    b = int(rng.integers(0, n))
    return lambda k: (k * a + b) % n


def _graph(case, rng):
    """Distinct triples (s, p, o), predicate by predicate."""
    n, preds, total = case["entities"], case["predicates"], case["triples"]
    w = np.arange(1, preds + 1, dtype=np.float64) ** -case["pred_zipf"]
    if case["hub"]:   # the five hub predicates hold 400/6,800 of the triples each
        w[:] = (1.0 - 5 / 17) / (preds - 5)
        w[:5] = 1 / 17
    counts = np.maximum(1, np.rint(total * w / w.sum())).astype(np.int64)
    parts = []
    for p in range(preds):
        fs, fo = _relabel(rng, n, case["subj_zipf"]), _relabel(rng, n, case["obj_zipf"])
        want, keys = int(counts[p]), np.zeros(0, dtype=np.int64)
        if case["hub"] and p < 5:
            for _ in range(2):
                hub = int(rng.integers(0, n))
                keys = np.union1d(keys, rng.permutation(n)[:case["hub"]].astype(np.int64) * n + hub)
        for _ in range(60):
            if len(keys) >= want:
                break
            k = (want - len(keys)) * 2 + 16
            s = fs(_zipf_ranks(rng, n, case["subj_zipf"], k))
            o = fo(_zipf_ranks(rng, n, case["obj_zipf"], k))
            fresh = np.setdiff1d(s.astype(np.int64) * n + o, keys)
            if len(keys) + len(fresh) > want:
                fresh = rng.permutation(fresh)[:want - len(keys)]
            keys = np.union1d(keys, fresh)
        parts.append(np.stack([keys // n, np.full(len(keys), p, dtype=np.int64), keys % n], axis=1))
    return np.concatenate(parts)


def _pick(rng, cum):
    return int(min(np.searchsorted(cum, rng.random() * cum[-1], side="right"), len(cum) - 1))


def _chain(rng, length, cum, hubs, i):
    """(?a .. ?v1) .. (?vk .. ?b) => (?a p ?b), each atom in a random direction."""
    names = ["?a"] + ["?v%d" % k for k in range(1, length)] + ["?b"]
    preds = [_pick(rng, cum) for _ in range(length)]
    dirs = [int(rng.integers(0, 2)) for _ in range(length)]
    if hubs:
        hub = int(rng.integers(0, 5))
        if i % 2 == 0:   # through a hub from both sides
            k = int(rng.integers(0, length - 1))
            preds[k] = preds[k + 1] = hub
            dirs[k], dirs[k + 1] = 0, 1
        else:
            preds[int(rng.integers(0, length))] = hub
    body = tuple((names[k], preds[k], names[k + 1]) if dirs[k] == 0 else (names[k + 1], preds[k], names[k])
                 for k in range(length))
    return ("?a", _pick(rng, cum), "?b"), body


def _mined(rng, lo, hi, cum):
    """A refinement of the miner: an atom on ?a or ?b, then dangling or closing atoms."""
    head = ("?a", _pick(rng, cum), "?b")
    q = _pick(rng, cum)
    first = [("?a", q, "?b"), ("?b", q, "?a"), ("?a", q, "?v0"), ("?v0", q, "?a"), ("?b", q, "?v0"), ("?v0", q, "?b")]
    first = [a for a in first if a != head]
    rule = miner.Rule(head, (first[int(rng.integers(0, len(first)))],))
    while len(rule.body) < hi and (len(rule.body) < lo or rng.random() < 0.5):
        more = miner.refinements(rule, [_pick(rng, cum)], 4)
        if not more:
            break
        rule = more[int(rng.integers(0, len(more)))]
    return rule.head, rule.body


def _rule_set(case, rng, triples):
    size = np.bincount(triples[:, 1], minlength=case["predicates"]).astype(np.float64)
    cum = np.cumsum(size if case["pred_zipf"] > 0 or case["hub"] else np.ones(case["predicates"]))
    lo, hi = case["min_atoms"], case["max_atoms"]
    if case["kind"] == "mined":
        return [_mined(rng, lo, hi, cum) for _ in range(case["rules"])]
    if case["pred_zipf"] > 0:   # the configuration's length weights
        w = np.cumsum(np.array([0.2, 0.4, 0.3, 0.1])[lo - 1:hi])
    elif case["call"] == "serve":   # geometric lengths
        w = np.cumsum(0.6 ** np.arange(lo - 1, hi))
    else:
        w = np.cumsum(np.ones(hi - lo + 1))
    hubs = {"hub": case["rules"], "biomedical": case["rules"] // 5}.get(case["kind"], 0)
    return [_chain(rng, max(lo + _pick(rng, w), 2 if i < hubs else 1), cum, i < hubs, i) for i in range(case["rules"])]


def _text(rule):
    head, body = rule
    atom = lambda a: "(%s <http://p/%d> %s)" % a   # noqa: E731
    return " ^ ".join(map(atom, body)) + " => " + atom(head)


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 2])
    triples = _graph(case, rng)
    return triples, _rule_set(case, rng, triples)


def prepare(case, seed):
    triples, rules = _inputs(case, seed)
    fd, path = tempfile.mkstemp(suffix=".ttl")
    try:
        with os.fdopen(fd, "w") as f:
            f.write("".join(["<http://e/%d> <http://p/%d> <http://e/%d> .\n" % (s, p, o)
                             for s, p, o in triples.tolist()]))
        lib = eng.GpuRulesLib(path)
    finally:
        os.unlink(path)
    state = {"call": case["call"], "lib": lib, "rules": [_text(r) for r in rules]}
    if case["call"] == "replay":
        state["batch"] = lib.prepare_batch(state["rules"])
        state["batch"].autotune(3)
    elif case["call"] == "serve":
        state["server"] = lib.serve(slots=4)
    return state


# ---------------------------------------------------------------- the calls

def run(state):
    call, lib, rules = state["call"], state["lib"], state["rules"]
    if call == "each":
        got = [lib.evaluate_rule(r) for r in rules]
        return {f: np.array([getattr(g, f) for g in got]) for f in FIELDS}
    if call == "batch":
        results, status, _ = lib.evaluate_rules_batch(rules)
        a = np.frombuffer(results, dtype=RESULT)
        return dict({f: a[f] for f in FIELDS}, status=np.array(status))
    if call == "replay":
        state["batch"].run(fetch=False)
        return state["batch"].counts()
    server, n = state["server"], len(rules)
    for i, r in enumerate(rules):
        server.submit(i, r)
    out = np.zeros(n, dtype=RESULT)
    left = n
    while left:
        for i, status, g, _ in server.poll(wait_ms=20):
            if status != 0:
                raise RuntimeError("request %d: status %d" % (i, status))
            out[i] = (g.support, g.headSize, g.headSupport, g.headCoverage, g.bodySize, g.confidence, 0.0, 0.0)
            left -= 1
    return {f: out[f] for f in FIELDS}


def work(case):
    """Every triple of the predicates that the rules name read once (a subject
    and an object), each rule's text read and its result written."""
    atoms = case["rules"] * ((case["min_atoms"] + case["max_atoms"]) / 2 + 1)
    named = case["predicates"] * (1 - (1 - 1 / case["predicates"]) ** atoms)
    return {"bytes": 8.0 * case["triples"] * named / case["predicates"] + case["rules"] * 156.0, "flops": 0.0}


# ---------------------------------------------------------------- 64-bit values

class _TooLong(Exception):
    pass


class _Joins:
    """Rule counts by plain joins over sorted arrays."""

    def __init__(self, case, triples, limit):
        self.n = case["entities"]
        self.left = limit
        self.fwd, self.rev = {}, {}
        for p in range(case["predicates"]):
            t = triples[triples[:, 1] == p]
            self.fwd[p] = np.sort(t[:, 0] * self.n + t[:, 2])
            self.rev[p] = np.sort(t[:, 2] * self.n + t[:, 0])

    def rows(self, table, body):
        """All groundings of `body` that extend the bindings in `table` (variable -> column; 'root' -> index)."""
        todo = list(body)
        while todo:
            todo.sort(key=lambda a: -((a[0] in table) + (a[2] in table)))
            s, p, o = todo.pop(0)
            if s in table and o in table:
                k = table[s] * self.n + table[o]
                keep = np.zeros(len(k), dtype=bool)
                if len(self.fwd[p]):
                    at = np.minimum(np.searchsorted(self.fwd[p], k), len(self.fwd[p]) - 1)
                    keep = self.fwd[p][at] == k
                table = {v: c[keep] for v, c in table.items()}
                continue
            if s not in table and o not in table:
                raise _TooLong("no bound variable")
            edges, known, fresh = (self.fwd[p], s, o) if s in table else (self.rev[p], o, s)
            lo = np.searchsorted(edges, table[known] * self.n)
            cnt = np.searchsorted(edges, table[known] * self.n + self.n) - lo
            total = int(cnt.sum())
            self.left -= total
            if self.left < 0:
                raise _TooLong("too many bindings")
            rep = np.repeat(np.arange(len(cnt)), cnt)
            off = np.arange(total) - np.repeat(np.cumsum(cnt) - cnt, cnt)
            new = edges[lo[rep] + off] % self.n
            keep = np.ones(total, dtype=bool)
            for v, c in table.items():
                if v != "root":
                    keep &= c[rep] != new
            table = {v: c[rep[keep]] for v, c in table.items()}
            table[fresh] = new[keep]
        return table

    def counts(self, rule):
        """(support, head size, body size); head and body variables are distinct, so two atoms
        can only ground to one triple when they are the same atom."""
        head, body = rule
        hs, ho = self.fwd[head[1]] // self.n, self.fwd[head[1]] % self.n
        if len(set(body)) < len(body):
            return 0, len(hs), 0
        sup = 0
        if head not in body:
            ok = hs != ho
            t = self.rows({"root": np.flatnonzero(ok), head[0]: hs[ok], head[2]: ho[ok]}, body)
            sup = len(np.unique(t["root"]))
        seeds = [(self.fwd if a[0] == head[0] else self.rev)[a[1]] for a in body if head[0] in (a[0], a[2])]
        if not seeds:
            return sup, len(hs), 0
        first = np.unique(min(seeds, key=len) // self.n)
        t = self.rows({"root": np.arange(len(first)), head[0]: first}, body)
        pairs = t["root"] * self.n + t[head[2]] if head[2] in t else t["root"]
        return sup, len(hs), len(np.unique(pairs))


def exact(case, seed):
    triples, rules = _inputs(case, seed)
    joins = _Joins(case, triples, 30_000_000)
    try:
        c = np.array([joins.counts(r) for r in rules], dtype=np.int64)
    except _TooLong:
        return None
    sup, size, body = c[:, 0], c[:, 1], c[:, 2]
    if case["call"] == "replay":
        return np.stack([sup, size, size, body], axis=1)
    out = {"support": sup.astype(np.int32), "headSize": size.astype(np.int32), "headSupport": size.astype(np.int32),
           "headCoverage": np.where(size > 0, sup / np.maximum(size, 1), 0.0), "bodySize": body.astype(np.int32),
           "confidence": np.where(body > 0, sup / np.maximum(body, 1), 0.0)}
    return dict(out, status=np.zeros(len(rules), dtype=np.int64)) if case["call"] == "batch" else out
