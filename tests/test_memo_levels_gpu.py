"""Chains through hub rows against the C oracle, at the places where suffix
memos, claims and the choice of the root end can go wrong: hubs at every
level of 2- to 5-atom chains (a four-atom plan has a three-step memo at level
1 and a two-step memo at level 2), hubs that are their own neighbours, bound
values that are neighbours of the hub, and many paths to one hub row."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import terms_to_ir

pytestmark = pytest.mark.gpu

P_SPARSE, P_OUT, P_IN, P_HEAD = range(4)


@pytest.fixture(scope="module")
def hub_chains(tmp_path_factory):
    """Entities 0..5 are hubs, 6..125 the rest.  p0: rest -> any, out-degree
    1-2 (self-loops among them); p1: hub -> 40 of all, two hubs to themselves;
    p2: rest -> 1-3 hubs, two hubs to themselves; p3: head pairs.  48 seeded
    chains of 2-5 atoms.  Returns (ttl, rules, int64 counts [n, 4])."""
    import oracle
    rng = np.random.default_rng(3)
    hubs, every = np.arange(6), np.arange(126)
    rest = every[6:]
    trip = {(int(h), P_OUT, int(v)) for h in hubs for v in rng.choice(every, 40, replace=False)}
    trip |= {(h, P_OUT, h) for h in (0, 1)} | {(h, P_IN, h) for h in (1, 2)}
    for v in rest:
        trip |= {(int(v), P_SPARSE, int(w)) for w in rng.choice(every, rng.integers(1, 3), replace=False)}
        trip |= {(int(v), P_IN, int(h)) for h in rng.choice(hubs, rng.integers(1, 4), replace=False)}
        if v % 9 == 0:
            trip.add((int(v), P_SPARSE, int(v)))
    while sum(p == P_HEAD for _, p, _ in trip) < 700:
        trip.add((int(rng.choice(every)), P_HEAD, int(rng.choice(every))))
    rules, terms = [], []
    for i in range(48):
        m = 2 + i % 4
        names = ["a"] + [f"v{k}" for k in range(1, m)] + ["b"]
        body = []
        for k in range(m):
            x, y = names[k], names[k + 1]
            if rng.integers(0, 2):
                x, y = y, x
            body.append((int(rng.integers(0, 3)), ("v", x), ("v", y)))
        head = (P_HEAD, ("v", "a"), ("v", "b"))
        terms.append(body + [head])
        text = [f"(?{s[1]} <http://h/p{p}> ?{o[1]})" for p, s, o in terms[-1]]
        rules.append(" ^ ".join(text[:-1]) + " => " + text[-1])
    trip = np.array(sorted(trip), dtype=np.int32)
    ttl = tmp_path_factory.mktemp("hubs") / "hubs.ttl"
    ttl.write_text("".join(f"<http://h/e{s}> <http://h/p{p}> <http://h/e{o}> .\n" for s, p, o in trip.tolist()))
    g = oracle.OracleGraph(trip, P_HEAD + 1)
    counts, st = g.evaluate_ir(terms_to_ir(terms), len(rules))
    g.close()
    assert (st == 0).all()
    return ttl, rules, counts


@pytest.mark.parametrize("hub_min,gain", [("8", "0"), ("8", "0.25"), ("0", "0")])
@pytest.mark.parametrize("switch", ["", "GPU_RULES_MEMO3", "GPU_RULES_HUB_CLAIMS", "GPU_RULES_PLAN_BOTH_ENDS"])
def test_hub_chain_counts(hub_chains, hub_min, gain, switch, monkeypatch):
    ttl, rules, exp = hub_chains
    monkeypatch.setenv("GPU_RULES_HUB_MIN_DEGREE", hub_min)
    monkeypatch.setenv("GPU_RULES_MEMO_GAIN", gain)
    if switch:
        monkeypatch.setenv(switch, "0")
    with eng.GpuRulesLib(ttl) as lib:
        b = lib.prepare_batch(rules)
        b.run()
        got = b.counts()
        b.close()
        bad = [(rules[i], got[i].tolist(), exp[i].tolist()) for i in range(len(rules)) if not (got[i] == exp[i]).all()]
        assert not bad, f"{len(bad)} of {len(rules)} rules differ, first: {bad[:2]}"
        for i in range(0, len(rules), 5):
            r = lib.evaluate_rule(rules[i])
            assert [r.support, r.headSize, r.headSupport, r.bodySize] == exp[i].tolist(), rules[i]
