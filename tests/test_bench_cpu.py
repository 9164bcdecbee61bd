"""bench.py ends with its one line whatever happens to a leg or the reference."""
import json
import os
import pathlib
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).parents[1]


def test_a_leg_that_does_not_end():
    code = """
import time, bench
legs = {"first": {"value": 1}}
d = bench.LegDeadline({"metric": "m", "value": 2.0}, legs, 0.5)
d.start("first"); d.stop()
d.start("second")
time.sleep(60)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=50)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["value"] == 2.0 and line["legs"]["first"] == {"value": 1} and "did not end" in line["legs"]["second"]["error"]


@pytest.mark.parametrize("workload", ["config1", "config4"])
def test_reference_arm_without_the_reference(workload):
    from oracle.oracle import RefLib
    if RefLib.available():
        pytest.skip("the reference's library is built here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--workload", workload], cwd=ROOT,
                       capture_output=True, text=True, timeout=300, env=dict(os.environ))
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and "absent" in line["unavailable"]
