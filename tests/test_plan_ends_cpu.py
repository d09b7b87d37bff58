"""The planner's shared-memory layout for plans from either end and with row
scans of free variables, and that the plain plans have neither
(tests/native/plan_ends_check.cpp, compiled here with g++)."""
import re
import subprocess

import pytest

from conftest import ROOT, fuzz_names, load_fixture
from masterthesis_gpu_acceleration_b200 import synth

CSRC = ROOT / "masterthesis_gpu_acceleration_b200" / "csrc"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    out = tmp_path_factory.mktemp("native") / "plan_ends_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-o", str(out),
                    str(ROOT / "tests" / "native" / "plan_ends_check.cpp")] +
                   [str(CSRC / f) for f in ("turtle.cpp", "index.cpp", "rules.cpp", "planner.cpp", "tasks.cpp")],
                   check=True)
    return out


def _run(checker, ttl, rules):
    r = subprocess.run([str(checker), str(ttl), str(rules)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return [int(x) for x in re.findall(r"\d+", r.stdout)]


@pytest.mark.parametrize("name", fuzz_names() + ["edge_cases.json"])
def test_either_end_fixtures(checker, tmp_path, name):
    fx = load_fixture(name)
    ttl, rules = tmp_path / "graph.ttl", tmp_path / "rules.txt"
    ttl.write_text(fx["ttl"])
    texts = fx["rules"] if "rules" in fx else [c["rule"] for c in fx["cases"]]
    rules.write_text("\n".join(texts) + "\n")
    _run(checker, ttl, rules)


@pytest.mark.parametrize("cfg,n", [("c3", 2000), ("c4s", None)])
def test_either_end_synthetic(checker, data_dir, cfg, n):
    d = synth.generate(cfg, data_dir / f"{cfg}_ends", seed=0)
    texts = synth.read_rules(d)[:n]
    preds = sorted(set(re.findall(r"<[^>]*>", "\n".join(texts))))[:40]
    # a part that nothing reaches, with a free variable
    texts += [f"(?a {p} ?x) ^ (?b {q} ?y) => (?a {p} ?b)" for p, q in zip(preds, preds[1:])]
    rules = data_dir / f"{cfg}_ends" / "some.txt"
    rules.write_text("\n".join(texts) + "\n")
    phases, far, scans, _ = _run(checker, d / "graph.ttl", rules)
    assert phases > 0 and far > 0 and scans > 0
