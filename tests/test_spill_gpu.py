"""Spilled tasks (open frontier items given to follow-up launches) against the
reference's fixtures and the C oracle: every task spills after its first
round, and what it spilled spills once more, so records of every level, of
both phases, of split heavy roots and of global rows are resumed, up to lists
that are full (the task then runs on)."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import GOLDEN, fuzz_names, load_fixture
from masterthesis_gpu_acceleration_b200 import synth
from test_free_variables_gpu import free_rules   # noqa: F401  (fixture)
from test_memo_levels_gpu import hub_chains   # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

COUNT_FIELDS = ("support", "headSize", "headSupport", "bodySize")


def _check(ttl, rules, exp, options=()):
    with eng.GpuRulesLib(ttl) as lib:
        for name, value in options:
            lib.set_option(name, value)
        with lib.prepare_batch(rules) as b:
            for _ in range(2):
                b.run()
                got = b.counts()
                bad = [(rules[i], got[i].tolist(), exp[i].tolist()) for i in range(len(rules))
                       if not (got[i] == exp[i]).all()]
                assert not bad, f"{len(bad)} of {len(rules)} rules differ, first: {bad[:2]}"
        res, _, _ = lib.evaluate_rules_batch(rules)
        for i in range(0, len(rules), max(1, len(rules) // 20)):
            assert [getattr(res[i], f) for f in COUNT_FIELDS] == exp[i].tolist(), rules[i]
            r = lib.evaluate_rule(rules[i])
            assert [getattr(r, f) for f in COUNT_FIELDS] == exp[i].tolist(), rules[i]


@pytest.fixture(autouse=True)
def _always(monkeypatch):
    monkeypatch.setenv("GPU_RULES_SPILL", "2")


@pytest.mark.parametrize("name", fuzz_names())
def test_spill_fuzz(tmp_path, name):
    fx = load_fixture(name)
    p = tmp_path / "graph.ttl"
    p.write_text(fx["ttl"])
    exp = np.array([[e[k] for k in COUNT_FIELDS] for e in fx["expected"]], dtype=np.int64)
    _check(p, fx["rules"], exp)


@pytest.mark.parametrize("options", [(), (("task_target", 16),), (("dedup_mode", 1),), (("dedup_mode", 2),)])
@pytest.mark.parametrize("hub_min", ["0", "8"])
def test_spill_hub_chains(hub_chains, options, hub_min, monkeypatch):   # noqa: F811
    monkeypatch.setenv("GPU_RULES_HUB_MIN_DEGREE", hub_min)
    monkeypatch.setenv("GPU_RULES_MEMO_GAIN", "0")
    _check(*hub_chains, options)


def test_spill_free_variables(free_rules):   # noqa: F811
    _check(*free_rules)


def test_spill_dense_and_full_lists(data_dir):
    """Dense rules (long rounds) and 400 DBpedia-shaped ones: more records than
    a list holds."""
    for cfg, name, n in (("c2s", "synthetic_c2s.json", None), ("c3", None, 400)):
        d = synth.generate(cfg, data_dir / cfg, seed=0)
        rules = synth.read_rules(d)[:n]
        if name:
            exp = np.array([[e[k] for k in COUNT_FIELDS] for e in load_fixture(name)["expected"]], dtype=np.int64)
        else:
            with np.load(GOLDEN / "c3_seed0.npz") as z:
                exp = z["expected"][:n].astype(np.int64)
        _check(d / "graph.ttl", rules, exp)
