"""Two graphs served side by side under time limits (the DBpedia-like one and
the biomedical one, whose long chains through hubs take far longer than the
limits): requests expected above the limit are refused, so that the others do
not wait behind them, and what is answered is exact."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from masterthesis_gpu_acceleration_b200 import serving, synth

pytestmark = pytest.mark.gpu


def test_limits_keep_two_graphs_served(data_dir, tmp_path):
    """5,000 requests/s for 1.5 s, half of them to each graph, after half a
    second at 1,000: at least 4,500/s are completed, half of the first graph's
    within 20 ms (the limit), no request is left without an answer."""
    graphs = []
    try:
        for g, cfg in enumerate(("c3", "c4")):
            d = synth.generate(cfg, data_dir / cfg, seed=0)
            n_pred = int(synth.read_meta(d)["predicates"])
            pc = synth.pred_counts(synth.read_triples(d), n_pred)
            stream = synth.rule_stream(pc, 4000, tmp_path / cfg, p=0.4, max_len=8, seed=1 + g)
            lib = eng.GpuRulesLib(d / "graph.ttl")
            graphs.append((lib, synth.read_rules(stream)))
            lib.set_option("serve_deadline_us", 200000)
            lib.set_option("serve_max_us", 20000)
        serving.run_rate_multi(graphs, 1000, 0.5, seed=5)
        row, res = serving.run_rate_multi(graphs, 5000, 1.5, seed=6)
        assert {v[1] for r in res for v in r.values()} <= {0, -4}
        assert row["completed_ok"] + row["shed_over_time_limits"] == row["submitted"]
        assert row["sustained_rules_per_s"] >= 4500, row
        assert row["per_graph"][0]["p50_ms"] < 20, row
        rng = np.random.default_rng(3)
        for (lib, rules), r in zip(graphs, res):
            done = [v for v in r.values() if v[1] == 0]
            for i in rng.choice(len(done), min(20, len(done)), replace=False):
                ri, _, got = done[int(i)]
                alone = lib.evaluate_rule(rules[ri])
                assert [got.support, got.bodySize] == [alone.support, alone.bodySize], rules[ri]
    finally:
        for lib, _ in graphs:
            lib.close()
