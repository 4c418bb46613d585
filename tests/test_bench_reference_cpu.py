"""bench.py --impl reference: a rate only from the reference itself, a line that says
so where its build is missing."""
import json
import os
import subprocess
import sys

import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(tmp_path, body):
    code = "import sys; sys.argv = ['bench.py', '--impl', 'reference', '--scale', '0.001']\n" \
           "sys.path[:0] = [%r, %r]\nimport oracle, bench\n%s\nbench.main()" % (ROOT, os.path.join(ROOT, "oracle"), body)
    r = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_no_build_no_rate(tmp_path):
    line = run(tmp_path, "oracle.ref_available = lambda: False")
    assert line["impl"] == "reference" and "value" not in line
    assert "not here" in line["unavailable"] and "\n" not in line["unavailable"]


def test_a_build_is_timed(tmp_path):
    """Any command line with the reference's interface, here the oracle's, in its place."""
    if not os.path.exists(O.CLI):
        O.build()
    line = run(tmp_path, "oracle.ref_available = lambda: True\noracle.REF = oracle.CLI")
    assert line["impl"] == "reference" and line["value"] > 0
    assert line["cpu_baseline"]["kind"] == "reference"
