"""Tables off the TMA path, compiled at their first application (the tests of
test_gpu_generic_points.py with psb_set_generic_compile(1): by default their few
applications would be interpreted), and the default: a table's first applications
do not wait for the compiler, and the run that brings it to eight takes the compiled
kernel, with the same bits before, then and in replayed graphs."""
import os
import subprocess
import sys

import numpy as np
import pytest

import physis_b200 as ps
from tests import gpu_util as U
from tests import test_gpu_generic_points as P

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def compiled():
    ps.PSInit()
    ps.set_generic_compile(True)


@pytest.mark.parametrize("layout", sorted(U.LAYOUTS))
@pytest.mark.parametrize("colored", [False, True], ids=["all", "redblack"])
@pytest.mark.parametrize("size", [0, 1, 2])
@pytest.mark.parametrize("nd", [1, 2, 3])
def test_compiled_points_equal_interpreted(compiled, nd, size, colored, layout):
    P.test_compiled_points_equal_interpreted(nd, size, colored, layout)


def test_rows_of_a_red_black_pass_replayed_from_a_graph(compiled):
    P.test_rows_of_a_red_black_pass_replayed_from_a_graph()


# Twelve terms with offsets that keep a table off the TMA path; `k` makes the
# table's shape a new one. Times are minima over five tables, so that a stall of
# the machine does not count.
CODE = """
import time
import numpy as np
import physis_b200 as ps
from tests import gpu_util as U
ps.PSInit()
n = 32
f = np.random.default_rng(6).random((n, n, n), dtype=np.float32)
d = ps.PSDomain3DNew(*(0, n) * 3)

def table(k):
    terms = [(ps.const(0.01 * (i + 1)), ps.get(0, (i % 5 - 7 - k, i % 3, -i), ps.BOUNDARY_PERIODIC))
             for i in range(12)]
    st = ps.GenericStencil(3, [(ps.PS_FLOAT, (0, 1, 2))] * 2, 1, ps.PS_FLOAT, terms)
    a, b = ps.PSGrid3DFloatNew(n, n, n), ps.PSGrid3DFloatNew(n, n, n)
    ps.PSGridCopyin(a, f)
    ps.sync()
    return a, b, ps.PSStencilMap(st.kernel_id, d, a, b), ps.PSStencilMap(st.kernel_id, d, b, a)

first, eighth = [], []
for k in range(6):
    a, b, ab, ba = table(k)
    t = [time.perf_counter()]
    for i in range(8):
        ps.PSStencilRun(ab if i % 2 == 0 else ba, 1)
        ps.sync()
        t.append(time.perf_counter())
    if k:
        first.append(max(t[i + 1] - t[i] for i in range(7)))
        eighth.append(t[8] - t[7])
print("first", min(first), "eighth", min(eighth))

# Runs of three pairs: single applications and a graph, interpreted until the third.
a, b, ab, ba = table(50)
got = []
for _ in range(4):
    ps.PSStencilRun(ab, ba, 3)
    got.append((ps.PSGridCopyout(a), ps.PSGridCopyout(b)))
ps.set_impl(ps.IMPL_GENERIC)
ps.PSGridCopyin(a, f)
for k in range(4):
    ps.PSStencilRun(ab, ba, 3)
    assert U.bits_equal(got[k][0], ps.PSGridCopyout(a)), k
    assert U.bits_equal(got[k][1], ps.PSGridCopyout(b)), k
print("equal")
"""


def test_first_applications_do_not_wait_for_the_compiler():
    env = {k: v for k, v in os.environ.items() if k != "PHYSIS_B200_GENERIC_COMPILE"}
    env["PYTHONPATH"] = ROOT
    r = subprocess.run([sys.executable, "-c", CODE], env=env, cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    words = r.stdout.split()
    first, eighth = float(words[1]), float(words[3])
    # Interpreting takes some tens of microseconds, the compiler tens of milliseconds.
    assert first < 0.01 and eighth > 0.01, r.stdout
    assert "equal" in words
