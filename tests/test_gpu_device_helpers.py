"""Device helpers of csrc/common.cuh, called alone through the kernels of tests/csrc/device_helpers.cu."""
import ctypes
import importlib.util
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def helpers(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("xtbeig_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc", "device_helpers.cu")
    out = str(tmp_path_factory.mktemp("helpers") / "device_helpers.so")
    subprocess.run([build.nvcc()] + build.ARCH + build.FLAGS + ["-I", build.CSRC, "-shared", "-o", out, src], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("raise_to,want,ends", [(2, 2, True), (7, 2, True), (1, 2, False)])
def test_wait_count(helpers, raise_to, want, ends):
    """A count that is never reached ends by the time limit (20 ms) with the timeout status, never in silence."""
    status, result = np.zeros(4, np.int32), np.zeros(32, np.int32)
    err = helpers.run_wait(raise_to, want, ctypes.c_longlong(20_000_000), status.ctypes.data_as(ctypes.c_void_p),
                           result.ctypes.data_as(ctypes.c_void_p))
    assert err == 0
    assert np.array_equal(result, np.full(32, int(ends)))
    assert list(status[:3]) == ([0, 0, 0] if ends else [1, 0, 5])
