"""The benchmark's reference arm runs the reference's own sources or says that it cannot (CPU)."""
import argparse
import json
import os
import sys

import dms_ctypes

sys.path.insert(0, dms_ctypes.REPO)
import bench  # noqa: E402


def test_reference_arm_without_the_reference_build(monkeypatch, capsys):
    """It does not time the C oracle in its place."""
    def no_pool(cores):
        raise AssertionError("workers started for %s" % bench.cpu_kind())

    monkeypatch.setattr(dms_ctypes, "REF_LIB", os.path.join(dms_ctypes.REPO, "oracle", "_ref", "no_such_build.so"))
    monkeypatch.setattr(bench, "cpu_pool", no_pool)
    monkeypatch.delenv("RANK", raising=False)
    bench.run_reference_arm(argparse.Namespace(gpus=1, steps=2, warmup=3, impl="reference"))
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
