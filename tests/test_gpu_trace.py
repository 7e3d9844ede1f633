"""With tracing on every PSStencilRun prints one line with its time, whichever
way the run took: passes of several steps, two Himeno sweeps per pass, single
steps (runtime/libphysis_rt_cuda.cc prints it for every run)."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import physis_b200 as ps
from tests import gpu_util as U
ps.PSInit()
n = 128
a, b = ps.PSGrid3DFloatNew(n, n, n), ps.PSGrid3DFloatNew(n, n, n)
d = ps.PSDomain3DNew(0, n, 0, n, 0, n)
m1 = ps.PSStencilMap(ps.DIFFUSION7, d, a, b, *[0.1] * 7)
m2 = ps.PSStencilMap(ps.DIFFUSION7, d, b, a, *[0.1] * 7)
ps.PSStencilRun(m1, m2, 10)
print("launches", ps.last_run_stats()[1])
gs = [ps.grid_new(ps.PS_FLOAT, (40, 30, 20)) for _ in range(14)]
d = ps.PSDomain3DNew(1, 39, 1, 29, 1, 19)
ps.PSStencilRun(ps.PSStencilMap(ps.HIMENO19, d, *gs, 0.8),
                ps.PSStencilMap(ps.HIMENO19, d, gs[1], gs[0], *gs[2:], 0.8), 4)
print("launches", ps.last_run_stats()[1])
ps.PSStencilRun(m1, 3)
print("launches", ps.last_run_stats()[1])
"""


def test_every_kind_of_run_prints_its_time():
    env = dict(os.environ, PHYSIS_B200_TRACE="1", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CODE], env=env, cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    launches = [int(v) for v in re.findall(r"launches (\d+)", r.stdout)]
    assert launches[0] < 20 and launches[1] < 8 and launches[2] == 3, launches
    assert len(re.findall(r"Stencil finished \(time: [0-9.]+\)", r.stderr)) == 3, r.stderr
