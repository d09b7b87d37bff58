"""Phase times of per-rule calls that spill: each phase's time holds the
launches that ran what it gave away.  With every task spilling after its first
round nearly all work lies in those launches, so a rule's support takes about
the share of its time that it takes without spilling."""
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from masterthesis_gpu_acceleration_b200 import synth

pytestmark = pytest.mark.gpu


def test_phase_times_with_spilling(data_dir, monkeypatch):
    monkeypatch.setenv("GPU_RULES_FUSE_SUPPORT", "0")   # two phases, two launches
    d = synth.generate("c2s", data_dir / "c2s", seed=0)
    rules = synth.read_rules(d)
    share = {}
    for mode in ("0", "2"):
        monkeypatch.setenv("GPU_RULES_SPILL", mode)
        with eng.GpuRulesLib(d / "graph.ttl") as lib:
            for r in rules:
                lib.evaluate_rule(r)
            res = [lib.evaluate_rule(r) for r in rules]
            share[mode] = [r.supportMs / (r.supportMs + r.confidenceMs) for r in res]
    heavy = [i for i, x in enumerate(share["0"]) if x > 0.4]
    assert heavy
    for i in heavy:
        assert share["2"][i] > 0.5 * share["0"][i], (rules[i], share["0"][i], share["2"][i])
