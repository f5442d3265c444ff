"""The reference arm of bench.py runs the compiled reference or says why not."""
import json
import sys

import bench
import oracle


def _arm(monkeypatch, capsys):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"])
    monkeypatch.delenv("RANK", raising=False)
    bench.main()
    return json.loads(capsys.readouterr().out.strip().splitlines()[-1])


def test_without_the_reference_it_is_unavailable(monkeypatch, capsys):
    monkeypatch.setattr(oracle, "have_ref", lambda: False)

    def refuse(*a, **k):
        raise AssertionError("the oracle was timed as the reference")

    monkeypatch.setattr(oracle, "port_mpn_mul", refuse)
    line = _arm(monkeypatch, capsys)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_with_the_reference_it_is_timed(monkeypatch, capsys):
    monkeypatch.setattr(oracle, "have_ref", lambda: True)
    timed = {"value": 1.0, "ms_per_step": 2.0, "unit": "Gbit/s", "cores": 1, "kind": "reference", "sample": "",
             "cpu_model": "", "gmp_version": ""}
    monkeypatch.setattr(bench, "cpu_baseline_run", lambda *a, **k: timed)
    line = _arm(monkeypatch, capsys)
    assert line["value"] == 1.0 and line["cpu_baseline"]["kind"] == "reference"
