"""What destroyed handles leave for the next one, on the GPU: given back on
request, and not met again after a device reset."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, molecule_case

pytestmark = pytest.mark.gpu


def test_release_cache_returns_the_memory(gpu_lib):
    import tabipb
    import torch

    tabipb.release_cache()
    free0 = torch.cuda.mem_get_info()[0]
    case = molecule_case(400, 11.0, 6.0, seed=6)

    def solve():
        with tabipb.TabiSolver(maxparnode=500) as s:
            b = s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                              case["atmchr"])[3]
            s.build_tree()
            return s.dgmres(s.permute(bvct=b)[3])["x"]

    x = solve()
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert kept > 64 << 20  # the leaf factors of 20,000 faces and more
    tabipb.release_cache()
    # what stays: modules that the solve loaded
    assert free0 - torch.cuda.mem_get_info()[0] < 32 << 20
    np.testing.assert_array_equal(solve(), x)
    # a live handle keeps its own
    with tabipb.TabiSolver(maxparnode=500) as s:
        s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                      case["atmchr"])
        tabipb.release_cache()
        s.build_tree()
        v = np.random.default_rng(0).normal(size=2 * s.nface)
        y = s.matvec(v)
        tabipb.release_cache()
        np.testing.assert_array_equal(s.matvec(v), y)


RESET = """
import ctypes as C
import sys
sys.path[:0] = [{pkg!r}, {tests!r}]
import numpy as np
import tabipb
from conftest import molecule_case
tabipb.load()
rt, drv = C.CDLL("libcudart.so.12"), C.CDLL("libcuda.so.1")
case = molecule_case(60, 6.0, 2.0, seed=1)

def context():
    c = C.c_ulonglong()
    assert drv.cuCtxGetId(None, C.byref(c)) == 0
    return c.value

def solve():
    with tabipb.TabiSolver(maxparnode=200) as s:
        b = s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                          case["atmchr"])[3]
        s.build_tree()
        r = s.dgmres(s.permute(bvct=b)[3])
        return r["x"], s.energy(case["chrpos"], case["atmchr"], r["x"])[0], context()

first = solve()
for k in range(2):
    assert rt.cudaDeviceReset() == 0
    assert rt.cudaFree(None) == 0
    # no launch unless the new context is told from the old one
    assert context() != first[2]
    again = solve()
    assert np.array_equal(again[0], first[0]) and again[1] == first[1]
print("ok")
"""


def test_handles_after_a_device_reset(gpu_lib):
    code = RESET.format(pkg=os.path.join(ROOT, "tabi-pb_b200"),
                        tests=os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=200,
                       cwd=ROOT)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
