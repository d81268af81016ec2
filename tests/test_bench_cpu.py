"""bench.py on a machine without the compiled reference: the reference arm says
so in its one line and ends well, and the GPU arm's cpu_baseline is that line
instead of an exception after minutes of GPU work."""
import json
import os
import subprocess
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def no_reference(monkeypatch, tmp_path):
    """the compiled reference at a path that does not exist"""
    import oracle

    monkeypatch.setattr(oracle.Reference.__init__, "__defaults__",
                        (str(tmp_path / "libmctdhb_ref.so"),))
    sys.path.insert(0, REPO)
    import bench

    return bench


def test_reference_arm_without_the_reference(no_reference, capsys):
    args = type("A", (), {"gpus": 1, "steps": 2, "warmup": 3})
    no_reference.run_reference(args)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and set(line) == {"impl", "unavailable"}
    assert "\n" not in line["unavailable"] and "libmctdhb_ref.so" in line["unavailable"]
    no_reference.run_reference_full_mix(args)
    assert "unavailable" in json.loads(capsys.readouterr().out)


def test_cpu_baseline_without_the_reference(no_reference):
    out = no_reference.cpu_sample([])
    assert list(out) == ["unavailable"] and "libmctdhb_ref.so" in out["unavailable"]
    json.dumps({"cpu_baseline": out})


def test_unreadable_library(monkeypatch, tmp_path, capsys):
    """a file that is no library"""
    import oracle

    bad = tmp_path / "libmctdhb_ref.so"
    bad.write_bytes(b"no library")
    monkeypatch.setattr(oracle.Reference.__init__, "__defaults__", (str(bad),))
    sys.path.insert(0, REPO)
    import bench

    assert list(bench.cpu_sample([])) == ["unavailable"]


def test_reference_arm_as_a_program():
    if os.path.exists(os.path.join(REPO, "oracle", "_ref", "libmctdhb_ref.so")):
        pytest.skip("compiled reference on this machine")
    r = subprocess.run([sys.executable, os.path.join(REPO, "bench.py"), "--impl", "reference",
                        "--gpus", "1", "--steps", "1", "--warmup", "3"], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and "unavailable" in line
