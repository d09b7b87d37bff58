"""Prepared batches spill only where tuning measured that it pays: a batch that
was not tuned, or of short tasks, takes no launches and no memory for it, and
counts are the stored ones whichever way was kept."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import GOLDEN
from masterthesis_gpu_acceleration_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 10000])
def test_tuned_spilling(data_dir, n):
    d = synth.generate("c3", data_dir / "c3", seed=0)
    rules = synth.read_rules(d)[:n]
    with np.load(GOLDEN / "c3_seed0.npz") as z:
        exp = z["expected"][:n].astype(np.int64)
    with eng.GpuRulesLib(d / "graph.ttl") as lib:
        with lib.prepare_batch(rules) as b:
            # the engine alone (and the support kernel of split roots): no follow-ups
            assert b.info()["kernels_per_run"] <= 2
            for _ in range(2):
                b.autotune(1)
                for _ in range(5):
                    b.run()
                    assert (b.counts() == exp).all()
                if n == 40:
                    assert b.info()["kernels_per_run"] <= 2
