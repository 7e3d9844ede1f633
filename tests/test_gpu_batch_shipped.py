"""Sweeps per item of batch members with the shipped tune table (the other tests
run without it): the size bucket of 129 to 256 points a side holds cubes that are
faster with one sweep (144, 160) and with two (240, 256), so the library's own
rule decides there, and small buckets keep one."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import json
import physis_b200 as ps
ps.PSInit()
b, gs, sides = ps.Batch(), [], (96, 144, 160, 240, 256)
for n in sides:
    g = [ps.grid_new(ps.PS_FLOAT, (n, n, n)) for _ in range(14)]
    gs += g
    b.add(ps.HIMENO19, g, [0.8], 2)
b.run(0)
print(json.dumps([b.layout(i)["t_depth"] for i in range(len(sides))]))
"""


def test_sweeps_per_item_in_the_shipped_buckets(tmp_path):
    env = dict(os.environ, PHYSIS_B200_TUNE_SHIPPED="1", PYTHONPATH=ROOT,
               PHYSIS_B200_TUNE_CACHE=str(tmp_path / "tune.json"))
    r = subprocess.run([sys.executable, "-c", CODE], env=env, cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert json.loads(r.stdout.strip().splitlines()[-1]) == [1, 1, 1, 2, 2]
