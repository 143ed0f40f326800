"""cvx_device_status reports the checks of the last call on a stream, not of an earlier one, whatever kinds of
calls follow each other (tests/device_status.cu, built with the library's own objects)."""
import os
import subprocess

import pytest

import __graft_entry__

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_errors_belong_to_the_last_call(tmp_path):
    b = __graft_entry__._load("cuda_voxelizer_gb300/build.py", "_cvx_build_for_test")
    objects = [os.path.join(b.OUT_DIR, s + ".o") for s in b.SOURCES if s != "api.cu"]
    exe = str(tmp_path / "device_status")
    subprocess.run([b.nvcc_path()] + b._flags() + ["-cudart", "shared", "-o", exe, os.path.join(ROOT, "tests", "device_status.cu")] +
                   objects, check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-4000:]
