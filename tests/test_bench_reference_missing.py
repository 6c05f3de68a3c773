"""The benchmark's reference arm where the compiled reference is missing: one
line that says so, with none of this library's code in the process."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
import argparse, sys
sys.path.insert(0, {root!r})
import bench
from oracle import refdump
refdump.have_ref = lambda *a, **k: False
bench.NX, bench.NY = 40, 10
bench.run_reference_arm(argparse.Namespace(steps=2, warmup=1), 0, 1)
maps = open("/proc/self/maps").read()
print("libccfd" in maps or any(k.split(".")[0] == "ccfd_b200" for k in sys.modules))
"""


def test_missing_reference_is_reported_and_replaced_by_nothing():
    r = subprocess.run([sys.executable, "-c", PROBE.format(root=ROOT)], capture_output=True, text=True,
                       timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    line, loaded = r.stdout.strip().splitlines()
    got = json.loads(line)
    assert got["impl"] == "reference" and got["unavailable"] and set(got) == {"impl", "unavailable"}
    assert loaded == "False"
