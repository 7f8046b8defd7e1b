"""bench.py's reference arm: the reference cannot be installed here, so the arm says so in one line and exits 0, whatever
the number of GPUs it is asked for, and times nothing of this repository in its place."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT


@pytest.mark.parametrize("rank", [None, "0", "1"])
def test_reference_arm_says_it_is_unavailable(rank):
    env = {k: v for k, v in os.environ.items() if k != "RANK"}
    if rank is not None:
        env["RANK"] = rank
    r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--gpus", "1", "--steps", "2",
                        "--warmup", "1"], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = [json.loads(line) for line in r.stdout.splitlines() if line.strip()]
    if rank == "1":
        assert lines == []
        return
    assert len(lines) == 1 and lines[0]["impl"] == "reference" and lines[0]["unavailable"]
    assert "value" not in lines[0]
