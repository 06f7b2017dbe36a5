"""Where the reference library cannot be compiled (its sources are not there),
bench.py's reference arm says so in one line and succeeds, and the oracle still
builds its restatement."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys
sys.path.insert(0, {root!r} + "/oracle")
import oracle
oracle.REF_SO, oracle.REF_SRC = {so!r}, {src!r}
{then}
"""


def run(tmp_path, then, *args):
    code = CODE.format(root=ROOT, so=str(tmp_path / "none.so"), src=str(tmp_path), then=then)
    return subprocess.run([sys.executable, "-c", code, *args], cwd=ROOT, capture_output=True,
                          text=True, timeout=300)


@pytest.mark.parametrize("workload", ["c2-sqexp", "c4-batch"])
def test_reference_arm_says_that_it_is_unavailable(tmp_path, workload):
    r = run(tmp_path, "sys.path.insert(0, '.'); import bench; bench.main()", "--impl",
            "reference", "--steps", "1", "--warmup", "0", "--workload", workload)
    assert r.returncode == 0, r.stderr[-1000:]
    lines = [json.loads(x) for x in r.stdout.splitlines() if x.startswith("{")]
    assert len(lines) == 1 and lines[0]["impl"] == "reference" and lines[0]["unavailable"]


def test_oracle_builds_without_the_sources(tmp_path):
    r = run(tmp_path, "oracle.build(); oracle.Oracle()")
    assert r.returncode == 0, r.stderr[-1000:]
