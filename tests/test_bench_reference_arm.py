"""bench.py --impl reference without jclsquant's own kernels: one line that says so, and no number from this
repository's restatement in its place."""
import json
import subprocess
import sys

from conftest import ROOT

CODE = """
import sys
sys.argv = ["bench.py", "--impl", "reference", "--cells", "6", "--M", "8", "--steps", "1", "--warmup", "3"]
import bench
bench.cpu_reference_kernels = lambda: None
bench.run_reference_arm(bench.parse())
"""


def test_unavailable_without_the_reference_kernels():
    out = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, stdout=subprocess.PIPE, text=True, check=True, timeout=120).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
