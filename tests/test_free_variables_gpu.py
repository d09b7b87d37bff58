"""Rules with variables that occur once (free variables) and with body parts
that share no variable with the rest, against the C oracle: rows shorter
than, as long as and longer than the rule's number of variables, self-loops,
bound values among a free variable's values, two free variables on one key,
row scans behind one and two bound values, and constants."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import terms_to_ir

pytestmark = pytest.mark.gpu

N, P_HEAD = 40, 3


def _text(atoms):
    t = lambda x: f"?{x[1]}" if x[0] == "v" else f"<http://f/e{x[1]}>"   # noqa: E731
    text = [f"({t(s)} <http://f/p{p}> {t(o)})" for p, s, o in atoms]
    return " ^ ".join(text[:-1]) + " => " + text[-1]


@pytest.fixture(scope="module")
def free_rules(tmp_path_factory):
    """40 entities, p0-p2 with out-degrees 0-8 (every fourth entity a
    self-loop), 160 head pairs; hand-written shapes and 120 seeded rules of
    1-4 atoms over ?a, ?b, up to three more variables and one constant."""
    import oracle
    rng = np.random.default_rng(17)
    trip = set()
    for p in range(3):
        for v in range(N):
            trip |= {(v, p, int(w)) for w in rng.choice(N, rng.integers(0, 9) if p else v % 4, replace=False)}
            if v % 4 == 0:
                trip.add((v, p, v))
    while sum(p == P_HEAD for _, p, _ in trip) < 160:
        trip.add((int(rng.integers(N)), P_HEAD, int(rng.integers(N))))
    v = lambda x: ("v", x)   # noqa: E731
    a, b, x, y, z = map(v, "abxyz")
    head = (P_HEAD, a, b)
    rules = [
        [(0, a, x), (1, b, y), head],                   # two parts, a free variable in each
        [(0, x, a), (1, y, b), head],
        [(0, a, x), (0, a, y), (0, a, b), head],        # two free variables on ?a's row
        [(1, a, x), (1, x, y), (2, b, z), head],        # a row scan behind two bound values
        [(1, a, x), (1, b, x), (2, b, z), head],        # a free variable behind ?b
        [(0, a, x), (1, b, y), (2, y, z), head],        # ... behind an inner variable
        [(0, a, x), (1, y, b), (1, b, y), head],        # a part without free variables
        [(1, a, x), (P_HEAD, a, y), head],              # ?b in no body atom
        [(1, b, x), head],                              # ?a in no body atom
        [(0, a, x), (1, b, y), (2, ("c", 3), z), head],  # a constant's row
        [(1, x, y), (0, a, b), head],                   # a part with neither end
    ]
    for _ in range(120):
        m = int(rng.integers(1, 5))
        terms = [a, b, x, y, z][:int(rng.integers(3, 6))]
        body = []
        for k in range(m):
            s, o = (terms[int(i)] for i in rng.choice(len(terms), 2, replace=False))
            if rng.random() < 0.05:
                o = ("c", int(rng.integers(N)))
            body.append((int(rng.integers(0, 4)) if rng.random() < 0.1 else int(rng.integers(0, 3)), s, o))
        rules.append(body + [head])
    trip = np.array(sorted(trip), dtype=np.int32)
    ttl = tmp_path_factory.mktemp("free") / "free.ttl"
    ttl.write_text("".join(f"<http://f/e{s}> <http://f/p{p}> <http://f/e{o}> .\n" for s, p, o in trip.tolist()))
    g = oracle.OracleGraph(trip, P_HEAD + 1)
    counts, st = g.evaluate_ir(terms_to_ir(rules), len(rules))
    g.close()
    assert (st == 0).all()
    return ttl, [_text(r) for r in rules], counts


@pytest.mark.parametrize("gain", ["-1", "0"])
@pytest.mark.parametrize("hub_min,ends", [("0", "1"), ("4", "1"), ("4", "0")])
def test_free_variable_counts(free_rules, gain, hub_min, ends, monkeypatch):
    ttl, rules, exp = free_rules
    monkeypatch.setenv("GPU_RULES_MEMO_GAIN", gain)
    monkeypatch.setenv("GPU_RULES_HUB_MIN_DEGREE", hub_min)
    monkeypatch.setenv("GPU_RULES_PLAN_BOTH_ENDS", ends)
    with eng.GpuRulesLib(ttl) as lib:
        for mode in (0, 3):
            lib.set_option("dedup_mode", mode)
            with lib.prepare_batch(rules) as batch:
                batch.run()
                got = batch.counts()
            bad = [(rules[i], got[i].tolist(), exp[i].tolist()) for i in range(len(rules))
                   if not (got[i] == exp[i]).all()]
            assert not bad, f"mode {mode}: {len(bad)} of {len(rules)} rules differ, first: {bad[:2]}"
        lib.set_option("dedup_mode", 0)
        for i in range(0, len(rules), 4):
            r = lib.evaluate_rule(rules[i])
            assert [r.support, r.headSize, r.headSupport, r.bodySize] == exp[i].tolist(), rules[i]
            r = lib.evaluate_rule_noalloc(rules[i])
            assert [r.support, r.headSize, r.headSupport, r.bodySize] == exp[i].tolist(), rules[i]
