"""A batch prepared with fused supports and staged again under another dedup
mode: the supports stay exact, whether the body-size rows then lie in shared
memory, one global row per root or per resident block, and whether tasks are
spilled (2: every one) or not (0)."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import fuzz_names, load_fixture
from test_memo_levels_gpu import hub_chains   # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

COUNT_FIELDS = ("support", "headSize", "headSupport", "bodySize")


def _check(ttl, rules, exp, mode):
    with eng.GpuRulesLib(ttl) as lib:
        with lib.prepare_batch(rules) as b:
            b.run()
            assert (b.counts() == exp).all()
            lib.set_option("dedup_mode", mode)
            b.autotune(1)
            for _ in range(2):
                b.run()
                got = b.counts()
                bad = [(rules[i], got[i].tolist(), exp[i].tolist()) for i in range(len(rules))
                       if not (got[i] == exp[i]).all()]
                assert not bad, f"{len(bad)} of {len(rules)} rules differ, first: {bad[:2]}"
            # keys hold no rows to count a support from: such plans keep theirs
            modes = set(b.dedup()[0].tolist())
            assert modes <= ({-1, 0, 3} if mode == 3 else {-1, mode}), modes


@pytest.mark.parametrize("spill", ["0", "2"])
@pytest.mark.parametrize("mode", [1, 2, 3])
def test_restaged_mode_keeps_fused_supports(tmp_path, hub_chains, monkeypatch, mode, spill):   # noqa: F811
    monkeypatch.setenv("GPU_RULES_SPILL", spill)
    _check(*hub_chains, mode)
    fx = load_fixture(fuzz_names()[0])
    p = tmp_path / "graph.ttl"
    p.write_text(fx["ttl"])
    _check(p, fx["rules"], np.array([[e[k] for k in COUNT_FIELDS] for e in fx["expected"]], dtype=np.int64), mode)
