"""Sort mode's distinct count against the C oracle, where its parts can go
wrong: no key and few keys, one and two radix passes, more plans than are
counted in shared memory, duplicates, and hash sets that overflow many times
over (each part is then taken by halves)."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import terms_to_ir

pytestmark = pytest.mark.gpu

N, PREDS = 1200, 9


@pytest.fixture(scope="module")
def paths(tmp_path_factory):
    """p0..p7: 8 random objects per entity; p8: one triple, whose object is
    only an object.  72 paths of two atoms: 64 give about 75,000 pairs each
    (4.9M keys, duplicates among them), 8 one or none."""
    import oracle
    rng = np.random.default_rng(11)
    trip = {(0, 8, N)}
    for p in range(8):
        trip |= {(s, p, int(o)) for s in range(N) for o in rng.choice(N, 8, replace=False)}
    pairs = [(a, b) for a in range(8) for b in range(8)] + [(8, b) for b in range(4)] + [(b, 8) for b in range(4)]
    terms = [[(a, ("v", "x"), ("v", "z")), (b, ("v", "z"), ("v", "y")), (i % 8, ("v", "x"), ("v", "y"))]
             for i, (a, b) in enumerate(pairs)]
    rules = []
    for t in terms:
        text = [f"(?{s[1]} <http://h/p{p}> ?{o[1]})" for p, s, o in t]
        rules.append(" ^ ".join(text[:-1]) + " => " + text[-1])
    trip = np.array(sorted(trip), dtype=np.int32)
    ttl = tmp_path_factory.mktemp("paths") / "paths.ttl"
    ttl.write_text("".join(f"<http://h/e{s}> <http://h/p{p}> <http://h/e{o}> .\n" for s, p, o in trip.tolist()))
    g = oracle.OracleGraph(trip, PREDS)
    counts, st = g.evaluate_ir(terms_to_ir(terms), len(rules))
    g.close()
    assert (st == 0).all()
    return ttl, rules, counts


@pytest.mark.parametrize("keys", ["", "16", "1000"])
def test_sort_parts(paths, keys, monkeypatch):
    ttl, rules, exp = paths
    if keys:
        monkeypatch.setenv("GPU_RULES_SORT_SET", keys)
    with eng.GpuRulesLib(ttl) as lib:
        lib.set_option("dedup_mode", 3)
        # every plan in one launch; a few large ones (one pass); the small ones
        for part in (slice(0, 72), slice(3, 9), slice(64, 72), slice(71, 72)):
            b = lib.prepare_batch(rules[part])
            for _ in range(2):
                b.run()
                got = b.counts()
                bad = np.nonzero((got != exp[part]).any(axis=1))[0]
                assert len(bad) == 0, (part, bad[:5].tolist(), got[bad[:3]].tolist(), exp[part][bad[:3]].tolist())
            assert set(b.dedup()[0].tolist()) <= {3, -1}
            b.close()
