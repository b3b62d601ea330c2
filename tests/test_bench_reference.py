"""bench.py and the reference's compiled library: it is built where the sources are before anything is
said to be missing, and where it stays missing the lines say why."""
import json
import subprocess
import sys

import pytest

import bench
from oracle import binding


def _main(monkeypatch, tmp_path, argv, build):
    monkeypatch.setattr(binding, "REF_SO", str(tmp_path / "libhns_ref.so"))
    monkeypatch.setattr(binding, "build", build)
    monkeypatch.setattr(sys, "argv", ["bench.py", *argv])
    ran = []
    for arm in ("reference_arm", "ours", "reference_arm_fire", "ours_fire", "box64_reference", "box64_ours"):
        monkeypatch.setattr(bench, arm, lambda args, *a, arm=arm: ran.append((arm, args)))
    bench.main()
    return ran


def _makes(path):
    return lambda ref=None: path.write_bytes(b"")


def _fails(ref=None):
    raise subprocess.CalledProcessError(2, "make")


def test_reference_arm_runs_where_the_library_can_be_built(monkeypatch, tmp_path):
    ran = _main(monkeypatch, tmp_path, ["--impl", "reference"], _makes(tmp_path / "libhns_ref.so"))
    assert [a for a, _ in ran] == ["reference_arm"]


@pytest.mark.parametrize("build", [lambda ref=None: None, _fails])
def test_reference_arm_says_why_it_cannot(monkeypatch, tmp_path, capsys, build):
    assert _main(monkeypatch, tmp_path, ["--impl", "reference"], build) == []
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libhns_ref.so" in line["unavailable"]


@pytest.mark.parametrize("argv", [[], ["--workload", "box64"], ["--workload", "fire1024"]])
def test_own_line_names_the_missing_baseline(monkeypatch, tmp_path, capsys, argv):
    (_, args), = _main(monkeypatch, tmp_path, argv, lambda ref=None: None)
    assert args.no_cpu_baseline
    bench.print_line({"details": {}, "cpu_baseline": None}, args)
    assert "libhns_ref.so" in json.loads(capsys.readouterr().out)["details"]["cpu_baseline"]
    (_, args), = _main(monkeypatch, tmp_path, [*argv, "--no-cpu-baseline"], _fails)
    bench.print_line({"details": {}}, args)
    assert json.loads(capsys.readouterr().out)["details"] == {}


def test_own_line_keeps_its_baseline_where_the_library_can_be_built(monkeypatch, tmp_path):
    (_, args), = _main(monkeypatch, tmp_path, [], _makes(tmp_path / "libhns_ref.so"))
    assert not args.no_cpu_baseline and args.cpu_unavailable is None
