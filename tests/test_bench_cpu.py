"""The benchmark on a machine without the reference's C core: the CPU baselines
of the MCMC section say so in their own entries, and the reference arm prints
its one line; neither ends the program."""
import json
import types

import bench
from oracle import oracle


def _no_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(oracle, "REF_SO", str(tmp_path / "libp4ref.so"))
    monkeypatch.setattr(oracle, "REF_COPY", str(tmp_path / "src"))
    monkeypatch.delenv(oracle.REF_ENV, raising=False)


def test_reference_core_says_why(monkeypatch, tmp_path):
    _no_reference(monkeypatch, tmp_path)
    assert "not on this machine" in bench.reference_core()


def test_baseline_without_the_core(monkeypatch, tmp_path):
    _no_reference(monkeypatch, tmp_path)
    why = bench.reference_core()
    assert bench.cpu_part(lambda: bench.cpu_chains("dna16", 1, 1, 1), why) == {"unavailable": why}


def test_baseline_that_fails_is_reported():
    def fails():
        raise RuntimeError("no core to run on")
    assert bench.cpu_part(lambda: {"gens_per_s": 2.0}, None) == {"gens_per_s": 2.0}
    assert "no core to run on" in bench.cpu_part(fails, None)["unavailable"]


def test_reference_arm_without_the_core(monkeypatch, tmp_path, capsys):
    _no_reference(monkeypatch, tmp_path)
    bench.reference_arm(types.SimpleNamespace(config="dna16", gpus=1, steps=1, warmup=1))
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "not on this machine" in line["unavailable"]
