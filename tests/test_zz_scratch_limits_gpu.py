"""Calls whose scratch is limited accept what they accepted when every rule was
planned from the head subject's end with edge scans: where the cheaper plan
needs more memory than the limit, the plain one is taken.

?b lies in a part of the body that nothing else reaches.  Its subjects under
p2 (390,000, each with a free object) are fewer than p3's or p5's edges
(391,000 each, from 20 subjects), so the row scan of p2 is cheaper than the
scan of p3, but binds ?b in a domain whose bitmap rows lie in global memory:
220 head subjects need 10.7 MB of the 8 MiB that gpu_evaluate_rule_noalloc
has, or of a server's budget.  From p3 the domain has 20 values."""
import time

import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng

pytestmark = pytest.mark.gpu

N_ROOT, N_KEY, N_P3 = 220, 390_000, 391_000
FIELDS = ("support", "headSize", "headSupport", "bodySize")


@pytest.fixture(scope="module")
def parts(tmp_path_factory):
    """p1: 220 head subjects to one object each; p2: 390,000 subjects to one or
    two objects; p3: 20 of those subjects (the first) to objects of their own, and
    p5 the same and 100 more; p4: 50 head pairs, half of them body pairs."""
    rng = np.random.default_rng(23)
    key0, obj0, o30, root0 = 0, 1_000_000, 2_000_000, 3_000_000
    rows = [(root0 + i, 1, root0 + 1000 + i) for i in range(N_ROOT)]
    keys = np.arange(N_KEY)
    rows += [(int(k), 2, obj0 + int(k)) for k in keys]
    rows += [(int(k), 2, obj0 + N_KEY + int(k)) for k in keys[:2000]]
    rows += [(int(i % 20), 3, o30 + i) for i in range(N_P3)]
    rows += [(int(i % 20), 5, o30 + i) for i in range(N_P3 + 100)]
    good = [(root0 + int(rng.integers(N_ROOT)), 4, int(i % 20)) for i in range(25)]
    rows += good + [(root0 + int(rng.integers(N_ROOT)), 4, 500 + i) for i in range(25)]
    rows = sorted(set(rows))
    ttl = tmp_path_factory.mktemp("parts") / "parts.ttl"
    ttl.write_text("".join(f"<http://s/e{s}> <http://s/p{p}> <http://s/e{o}> .\n" for s, p, o in rows))
    head = [(s, o) for s, p, o in rows if p == 4]
    # every (root, one of the 20) pair is a body pair
    sup = sum(o < 20 for _, o in head)
    return ttl, [sup, len(head), len(head), N_ROOT * 20]


RULE = ("(?a <http://s/p1> ?x) ^ (?b <http://s/p2> ?f) ^ (?b <http://s/p3> ?y) ^ "
        "(?b <http://s/p5> ?y) => (?a <http://s/p4> ?b)")


def test_noalloc_keeps_accepting(parts):
    ttl, exp = parts
    with eng.GpuRulesLib(ttl) as lib:
        r = lib.evaluate_rule(RULE)
        assert [getattr(r, f) for f in FIELDS] == exp
        for _ in range(2):
            r = lib.evaluate_rule_noalloc(RULE)
            assert [getattr(r, f) for f in FIELDS] == exp


def test_serving_keeps_accepting(parts):
    ttl, exp = parts
    with eng.GpuRulesLib(ttl) as lib:
        with lib.serve(slots=2, max_batch=4, mem_budget=4 << 20) as sv:
            sv.submit(7, RULE)
            got = []
            t0 = time.time()
            while not got and time.time() - t0 < 60:
                got = sv.poll(wait_ms=50)
    rid, status, r, _ = got[0]
    assert (rid, status) == (7, 0)
    assert [getattr(r, f) for f in FIELDS] == exp
