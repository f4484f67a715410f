"""The Fortran hooks stop, as on every other failure, when a reduction's bounded
wait ran out: no energy and no v1 is handed back."""
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = pathlib.Path(__file__).resolve().parent.parent

CHILD = """
import sys
from libcc_b200 import _native as N, api as A, synthetic as S
no, nu = 4, 17
inp = S.generate(no, nu, 3)
h = A.IjkGpuHooks(no, nu, inp.eh, inp.ep, inp.t2, inp.vm, inp.voe)
N.check(N.load().ccT_debug_wait_limit(None, int(sys.argv[1])), "limit")
for i in range(no):
    for j in range(i):
        for k in range(j):
            h.driver(i + 1, j + 1, k + 1, *[A.packed_columns(inp.vvvo, no, nu, x) for x in (i, j, k)])
h.finalize()
print("finalized")
"""


@pytest.mark.parametrize("limit", [-1, 0])
def test_finalize_reports_a_wait_that_ran_out(limit):
    r = subprocess.run([sys.executable, "-c", CHILD, str(limit)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    if limit < 0:  # the default limit: the hooks work
        assert r.returncode == 0 and "finalized" in r.stdout, r.stderr
    else:
        assert r.returncode == 1 and "finalized" not in r.stdout
        assert "ijk_gpu_finalize failed: device wait timed out" in r.stderr
