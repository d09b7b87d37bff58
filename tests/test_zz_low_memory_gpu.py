"""Calls on a device with little free memory: buffers that only save time (a
32 MB arena for suffix memos, 31 MB of spill lists) are taken smaller or done
without, and the counts are the stored ones."""
import numpy as np
import pytest

import masterthesis_gpu_acceleration_b200 as eng
from conftest import load_fixture
from masterthesis_gpu_acceleration_b200 import synth

pytestmark = pytest.mark.gpu

FREE = 26 << 20   # below either buffer


def test_little_free_memory(data_dir):
    import torch
    fx = load_fixture("synthetic_c4s.json")
    d = synth.generate("c4s", data_dir / "c4s", seed=fx["seed"])
    fields = ("support", "headSize", "headSupport", "bodySize")
    exp = np.array([[e[k] for k in fields] for e in fx["expected"]], dtype=np.int64)
    rules = fx["rules"] * 20   # enough work for a launch that may spill
    with eng.GpuRulesLib(d / "graph.ttl") as lib:
        lib.set_option("batch_chunks", 1)
        torch.cuda.synchronize()
        eaten = []
        try:
            for step in (1 << 30, 64 << 20, 2 << 20):
                while eng.query_vram()[0] >= FREE + step:
                    left = (eng.query_vram()[0] - FREE) // step * step
                    eaten.append(torch.empty(int(left), dtype=torch.uint8, device="cuda"))
            assert eng.query_vram()[0] < 32 << 20
            res, status, _ = lib.evaluate_rules_batch(rules)
            r = lib.evaluate_rule(rules[0])
        finally:
            eaten.clear()
            torch.cuda.empty_cache()
        got = np.array([[getattr(x, f) for f in fields] for x in res])
        assert (np.array(status) == 0).all() and (got == np.tile(exp, (20, 1))).all()
        assert [getattr(r, f) for f in fields] == exp[0].tolist()
