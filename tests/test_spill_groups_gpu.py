"""Tasks of several groups of roots in launches that spill, against the stored
counts: after each group a block goes on, gives the groups behind it away or
has given them away already.  Targets of about two groups (the last one alone
is left to give), of a few and of the most a task may hold; every task spills
after its first round (2) or once blocks are idle (1)."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import GOLDEN
from masterthesis_gpu_acceleration_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("target", [14000, 40000, 10**7])
@pytest.mark.parametrize("spill", ["1", "2"])
def test_spill_between_groups(data_dir, monkeypatch, spill, target):
    monkeypatch.setenv("GPU_RULES_SPILL", spill)
    d = synth.generate("c3", data_dir / "c3", seed=0)
    n = 600
    rules = synth.read_rules(d)[:n]
    with np.load(GOLDEN / "c3_seed0.npz") as z:
        exp = z["expected"][:n].astype(np.int64)
    with eng.GpuRulesLib(d / "graph.ttl") as lib:
        lib.set_option("task_target", target)
        with lib.prepare_batch(rules) as b:
            for _ in range(4):
                b.run()
                got = b.counts()
                bad = np.nonzero((got != exp).any(axis=1))[0]
                assert len(bad) == 0, f"rules {bad[:5].tolist()} differ"
