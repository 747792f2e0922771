"""A kernel launch that fails is an error of the call that made it, not a result.
The child process runs over a driver library that returns an error in place of
launching (tests/cpp/launch_errors.cpp); nothing of it reaches the GPU."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, sys
import numpy as np
shim = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
from vistio_b200 import api, _lib
pos = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0.2, 0.2, 0], [1, 1, 0], [0, 0.5, 0.1]], np.float32)
tris = np.array([[0, 1, 2], [3, 4, 5]], np.uint32)
for query in (api.broadphase_pairs, api.broadphase_pairs_noalloc):
    assert query(pos, tris, 0.1).tolist() == [[0, 1]]
    shim.fail_launches(1)
    try:
        found = query(pos, tris, 0.1)
    except _lib.VistioError as e:
        assert e.status == 6, e
    else:
        raise SystemExit("%s: %s for a launch that failed" % (query.__name__, found.tolist()))
    finally:
        shim.fail_launches(0)
    assert query(pos, tris, 0.1).tolist() == [[0, 1]]
print("ok")
"""

WHERE = """
import ctypes
ctypes.CDLL("libcuda.so.1")
print({line.split()[-1] for line in open("/proc/self/maps") if "/libcuda.so" in line}.pop())
"""


def test_broadphase_reports_a_failed_launch(tmp_path):
    real = subprocess.run([sys.executable, "-c", WHERE], capture_output=True, text=True, check=True).stdout.split()
    shim = str(tmp_path / "libcuda.so.1")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-soname,libcuda.so.1", "-o", shim,
                           os.path.join(ROOT, "tests", "cpp", "launch_errors.cpp"), "-ldl"])
    p = subprocess.run([sys.executable, "-c", CHILD, shim], cwd=ROOT, env=dict(os.environ, REAL_LIBCUDA=real[0], PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "ok" in p.stdout, p.stdout + p.stderr
