"""Three-step memo items whose root lies under several hubs, against the C
oracle: the values reached through the root are few, as many as are listed,
one more, and many, in all orientations of (?a)-(?v1)-(?v2)-(?v3)-(?b) over
one predicate."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import terms_to_ir

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [2, 13, 14, 15, 16, 60])
def test_roots_under_several_hubs(tmp_path, own):
    """p0: hubs 0 and 1 share half of their objects, hub 2 shares only object
    20 with them and has `own` objects of its own; entities 100.. have one to
    three objects.  p1: head pairs."""
    import oracle
    rng = np.random.default_rng(own)
    trip = {(0, 0, o) for o in range(20, 80)} | {(1, 0, o) for o in range(50, 110)}
    trip |= {(2, 0, 20)} | {(2, 0, 200 + k) for k in range(own)}
    for s in range(100, 160):
        trip |= {(s, 0, int(o)) for o in rng.choice(np.arange(20, 200 + own), 1 + s % 3, replace=False)}
    while sum(p == 1 for _, p, _ in trip) < 200:
        trip.add((int(rng.integers(20, 200)), 1, int(rng.integers(20, 200 + own))))
    terms, rules = [], []
    for bits in range(16):
        names = ["a", "v1", "v2", "v3", "b"]
        body = []
        for k in range(4):
            x, y = names[k], names[k + 1]
            if bits >> k & 1:
                x, y = y, x
            body.append((0, ("v", x), ("v", y)))
        t = body + [(1, ("v", "a"), ("v", "b"))]
        terms.append(t)
        text = [f"(?{s[1]} <http://h/p{p}> ?{o[1]})" for p, s, o in t]
        rules.append(" ^ ".join(text[:-1]) + " => " + text[-1])
    trip = np.array(sorted(trip), dtype=np.int32)
    ttl = tmp_path / "hubs.ttl"
    ttl.write_text("".join(f"<http://h/e{s}> <http://h/p{p}> <http://h/e{o}> .\n" for s, p, o in trip.tolist()))
    g = oracle.OracleGraph(trip, 2)
    exp, st = g.evaluate_ir(terms_to_ir(terms), len(rules))
    g.close()
    assert (st == 0).all()
    for env in ({}, {"GPU_RULES_PLAN_BOTH_ENDS": "0"}):
        with pytest.MonkeyPatch.context() as mp:
            mp.setenv("GPU_RULES_HUB_MIN_DEGREE", "8")
            mp.setenv("GPU_RULES_MEMO_GAIN", "0")
            for k, v in env.items():
                mp.setenv(k, v)
            with eng.GpuRulesLib(ttl) as lib:
                with lib.prepare_batch(rules) as b:
                    b.run()
                    got = b.counts()
        bad = np.nonzero((got != exp).any(axis=1))[0]
        assert len(bad) == 0, (env, [rules[i] for i in bad[:2]], got[bad[:2]].tolist(), exp[bad[:2]].tolist())
