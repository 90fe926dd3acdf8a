"""bench.py without a build of libuw12: the reference arm prints one line that says why and
ends normally, and the GPU arm is told the same reason instead of failing at the end."""
import argparse
import json

import bench
from oracle import ref_lib


def _without_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(ref_lib, "LIB_PATH", str(tmp_path / "ref.so"))
    monkeypatch.setattr(ref_lib, "TIMING_LIB_PATH", str(tmp_path / "timing.so"))
    monkeypatch.setattr(ref_lib, "REFERENCE_TREE", str(tmp_path))
    monkeypatch.setattr(ref_lib, "_libs", {})


def test_reference_arm_says_why(monkeypatch, tmp_path, capsys):
    _without_reference(monkeypatch, tmp_path)
    args = argparse.Namespace(config="c0", s_os=1.0, s_ss=0.5, steps=1, warmup=0, ref_rotation=1)
    bench.run_reference(args, 1, 2)  # other ranks print nothing
    assert capsys.readouterr().out == ""
    bench.run_reference(args, 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"]


def test_failed_build_is_a_reason(monkeypatch, tmp_path):
    _without_reference(monkeypatch, tmp_path)

    def fails(quiet=True):
        raise RuntimeError("reference build failed:\nerror: ...")
    monkeypatch.setattr(ref_lib, "build", fails)
    assert bench.cpu_reference_missing() == "reference build failed:"
