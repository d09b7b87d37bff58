"""The task builder's costs on CPU (tests/native/costs_check.cpp, compiled
here with g++), for rules planned from either end and tasks of several groups
of roots: they cover every root once, times that were learnt come back as the
expected times, and phases never run are expected in the units that tasks are
built in (the serving loop admits requests by these times).  Walks keep to
their budget, also where the second step is a free variable's and the
subjects are skewed, and rules that are small from either end are planned
without sampling the graph's transitions."""
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT, fuzz_names, load_fixture
from masterthesis_gpu_acceleration_b200 import synth

CSRC = ROOT / "masterthesis_gpu_acceleration_b200" / "csrc"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    out = tmp_path_factory.mktemp("native") / "costs_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-o", str(out),
                    str(ROOT / "tests" / "native" / "costs_check.cpp")] +
                   [str(CSRC / f) for f in ("turtle.cpp", "index.cpp", "rules.cpp", "planner.cpp", "tasks.cpp")],
                   check=True)
    return out


def _run(checker, ttl, rules):
    r = subprocess.run([str(checker), str(ttl), str(rules)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return [int(x) for x in re.findall(r"\d+", r.stdout)]


def test_costs_fixtures(checker, tmp_path):
    for name in fuzz_names() + ["edge_cases.json"]:
        fx = load_fixture(name)
        ttl, rules = tmp_path / f"{name}.ttl", tmp_path / f"{name}.txt"
        ttl.write_text(fx["ttl"])
        texts = fx["rules"] if "rules" in fx else [c["rule"] for c in fx["cases"]]
        rules.write_text("\n".join(texts) + "\n")
        _run(checker, ttl, rules)


@pytest.mark.parametrize("cfg,n", [("c2s", None), ("c4s", None), ("c3", 1500)])
def test_costs_synthetic(checker, data_dir, cfg, n):
    d = synth.generate(cfg, data_dir / f"{cfg}_costs", seed=0)
    rules = data_dir / f"{cfg}_costs" / "some.txt"
    rules.write_text("\n".join(synth.read_rules(d)[:n]) + "\n")
    phases, multi, split, unseen, *_, sampled, _, skew = _run(checker, d / "graph.ttl", rules)
    assert phases > 0 and unseen > 0
    assert sampled > 0 and skew >= 4000   # skewed or with hubs
    if cfg == "c3":
        assert multi > 0 and split > 0


def test_costs_free_second_step(checker, data_dir):
    """Dangling refinements of a skewed graph: ?f occurs once, behind ?x or ?b."""
    d = synth.generate("c3", data_dir / "c3_costs", seed=0)
    preds = sorted(set(re.findall(r"<[^>]*>", "\n".join(synth.read_rules(d)))))[::7]
    rules = data_dir / "c3_costs" / "free.txt"
    with open(rules, "w") as f:
        for i, p in enumerate(preds):
            q, h = preds[(i + 1) % len(preds)], preds[(i + 2) % len(preds)]
            f.write(f"(?a {p} ?x) ^ (?x {q} ?f) => (?a {h} ?b)\n")
            f.write(f"(?x {p} ?a) ^ (?f {q} ?x) => (?a {h} ?b)\n")
            f.write(f"(?a {p} ?b) ^ (?b {q} ?f) => (?a {h} ?b)\n")
            f.write(f"(?b {p} ?f) ^ (?a {q} ?x) => (?a {h} ?b)\n")
    assert _run(checker, d / "graph.ttl", rules)[0] > 0


def test_costs_uniform_graph(checker, tmp_path):
    """Chains of 4 to 8 atoms on a graph without skew."""
    rng = np.random.default_rng(5)
    ttl, rules = tmp_path / "uniform.ttl", tmp_path / "rules.txt"
    t = np.unique(np.stack([rng.integers(0, 10000, 100000), rng.integers(0, 20, 100000),
                            rng.integers(0, 10000, 100000)], axis=1), axis=0)
    ttl.write_text("".join(f"<http://u/e{s}> <http://u/p{p}> <http://u/e{o}> .\n" for s, p, o in t.tolist()))
    with open(rules, "w") as f:
        for i in range(60):
            names = ["a"] + [f"v{k}" for k in range(3 + i % 5)] + ["b"]
            atoms = []
            for x, y in zip(names, names[1:]):
                if rng.integers(0, 2):
                    x, y = y, x
                atoms.append(f"(?{x} <http://u/p{rng.integers(0, 20)}> ?{y})")
            f.write(" ^ ".join(atoms) + f" => (?a <http://u/p{rng.integers(0, 20)}> ?b)\n")
    phases, *_, sampled, _, skew = _run(checker, ttl, rules)
    # nor may a launch of them spill: no row is far longer than the others
    assert phases > 0 and sampled == 0 and skew < 4000
