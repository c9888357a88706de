"""bench.py prints its line whatever happens in the parts around the headline measurement: a part that raises reports
that in its key, one that never ends is given up at its limit with everything measured before it in the line, and the
reference arm says why it cannot run instead of failing."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import json, threading, time, bench
out = {}
parts = bench.Deadlines(out)
parts.start("headline", 30)
out.update({"value": 1.5, "first": None, "second": None, "third": None})
parts.ready = %s
parts.run("first", 30, lambda: {"x": 1})
parts.run("second", 30, lambda: 1 / 0)
%s
parts.run("third", 1, threading.Event().wait)
"""


def _child(ready, more=""):
    return subprocess.run([sys.executable, "-c", CHILD % (ready, more)], cwd=ROOT, capture_output=True, text=True,
                          timeout=120)


def test_a_part_that_does_not_end_keeps_the_line():
    r = _child(True)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["value"] == 1.5 and line["first"] == {"x": 1}
    assert "ZeroDivisionError" in line["second"]["error"]
    assert "did not end within 1 s" in line["third"]["error"]


def test_without_a_headline_there_is_no_line():
    r = _child(False)
    assert r.returncode == 1 and r.stdout == "" and "third did not end within 1 s" in r.stderr


@pytest.mark.skipif(os.path.exists(os.path.join(ROOT, "oracle", "_ref", "librans_ref.so")),
                    reason="the reference's coder is built: its arm runs")
def test_reference_arm_says_why_it_cannot_run():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "3"], cwd=ROOT,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and "librans_ref.so" in line["unavailable"]


def test_cpu_baseline_runs_without_the_references_coder():
    r = subprocess.run([sys.executable, "-c", "import json, bench; print(json.dumps(bench.cpu_baseline(128, 128, 1)))"],
                       cwd=ROOT, capture_output=True, text=True, timeout=200)
    assert r.returncode == 0, r.stderr
    out = json.loads(r.stdout)
    assert out["value"] > 0 and "rANS coder" in out["sample"]
