"""Slices of one rule evaluated by contexts that differ: their counts add up to
the whole rule's, whichever end each context plans its own calls from and
whatever it has evaluated before."""
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from test_memo_levels_gpu import hub_chains   # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def test_slices_of_different_contexts(hub_chains, monkeypatch):   # noqa: F811
    ttl, rules, exp = hub_chains
    monkeypatch.setenv("GPU_RULES_HUB_MIN_DEGREE", "8")
    monkeypatch.setenv("GPU_RULES_MEMO_GAIN", "0")
    libs = []
    for ends in ("1", "0"):
        monkeypatch.setenv("GPU_RULES_PLAN_BOTH_ENDS", ends)
        libs.append(eng.GpuRulesLib(ttl))
    try:
        libs[1].evaluate_rules_batch(rules)   # its memos exist before it cuts anything
        for n in (2, 3):
            for i, r in enumerate(rules):
                parts = [libs[k % 2].evaluate_rule_shard(r, k, n) for k in range(n)]
                got = [sum(p[0] for p in parts), parts[0][1], parts[0][2], sum(p[3] for p in parts)]
                assert got == exp[i].tolist(), (n, r)
    finally:
        for lib in libs:
            lib.close()
