"""bench.py's CPU leg: only a reference that is not there is reported as
unavailable; a baseline that is there and fails to build or run is an error."""
import json
import os

import pytest

import bench
import oracle
from oracle import stage_ref


def _fail(*args, **kwargs):
    raise FileNotFoundError("g++")


@pytest.fixture
def nothing(monkeypatch, tmp_path):
    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    monkeypatch.setattr(stage_ref, "DEST", str(tmp_path))
    monkeypatch.setattr(stage_ref, "reference_root", lambda: None)
    monkeypatch.setattr(bench, "run_reference_sample", _fail)
    return tmp_path


def test_without_the_reference_the_line_says_so(nothing):
    cpu = bench.cpu_baseline(None, [], 1, 1, 1.0, 1)
    assert cpu["value"] is None and "sources" in cpu["unavailable"]


@pytest.mark.parametrize("have", ["library", "staged", "checkout"])
def test_a_failing_baseline_is_not_an_absent_one(nothing, monkeypatch, have):
    if have == "library":
        monkeypatch.setattr(oracle, "ref_available", lambda: True)
    elif have == "staged":
        os.makedirs(nothing / "src")
    else:
        monkeypatch.setattr(stage_ref, "reference_root", lambda: str(nothing))
    with pytest.raises(FileNotFoundError, match="g\\+\\+"):
        bench.cpu_baseline(None, [], 1, 1, 1.0, 1)


def test_the_reference_arm_prints_its_line_without_the_reference(nothing, monkeypatch, capsys):
    monkeypatch.setattr("sys.argv", ["bench.py", "--impl", "reference", "--worlds", "2", "--steps", "1", "--warmup", "1"])
    bench.main()
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "sources" in line["unavailable"]
