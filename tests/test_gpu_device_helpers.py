"""Device helpers of csrc/common.cuh and internal stages, called alone through tests/csrc/device_helpers.cu."""
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
    subprocess.run([build.nvcc()] + build.ARCH + build.FLAGS + ["-I", build.CSRC, "-shared", "-o", out, src, build.LIB,
                                                                "-Xlinker", "-rpath=" + PKG], check=True)
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


@pytest.mark.parametrize("case", ["unit", "secular", "wide", "near_powers", "negative"])
def test_branch_free_division(helpers, case):
    """rcp_normal and div_normal against extended precision: half an ulp for the last rounding, and a hundredth for what
    precedes it (the cube of an approximation good to about 2^-20, and the residual's own correction).  Against the
    compiler's division, which rounds once: at most the neighbouring value."""
    import torch

    rng = np.random.default_rng(5)
    n = 1 << 18
    a, x = rng.uniform(1, 2, n), rng.uniform(1, 2, n)
    if case == "secular":  # z^2 over differences of poles
        a, x = 10.0 ** rng.uniform(-32, 0, n), 10.0 ** rng.uniform(-31, 0.3, n)
    elif case == "wide":
        a, x = np.ldexp(a, rng.integers(-400, 400, n)), np.ldexp(x, rng.integers(-400, 400, n))
    elif case == "near_powers":
        a = np.ldexp(1.0 + rng.integers(-64, 65, n) * 2.0**-52, rng.integers(-3, 4, n))
        x = np.ldexp(1.0 + rng.integers(-64, 65, n) * 2.0**-52, rng.integers(-3, 4, n))
    elif case == "negative":
        a, x = a * rng.choice([-1, 1], n), -x
    dev = [torch.from_numpy(v).cuda() for v in (a, x)] + [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    assert helpers.run_divide(n, *[ctypes.c_void_p(v.data_ptr()) for v in dev]) == 0
    rcp, quot, plain = (v.cpu().numpy() for v in dev[2:])
    al, xl = a.astype(np.longdouble), x.astype(np.longdouble)
    for got, exact in ((rcp, 1 / xl), (quot, al / xl)):
        # ulps of the exact value's binade (frexp: spacing on the lower side of a power of two is half as wide)
        ulp = np.ldexp(np.longdouble(1), np.frexp(exact)[1] - 53)
        assert (np.abs(got.astype(np.longdouble) - exact) / ulp).max() < 0.51
    assert np.abs(quot.view(np.int64) - plain.view(np.int64)).max() <= 1


def test_refused_gemm_launch_is_reported(helpers):
    """The launcher's own result is the only report of a launch that the runtime refuses: cudaErrorStreamCaptureImplicit."""
    assert helpers.run_refused_gemm(0) == 0  # nothing to launch
    assert helpers.run_refused_gemm(1) == 906


def _stedc(helpers, n, m_cols, code):
    import torch

    from oracle import inputs

    d, e = inputs.random_tridiagonal(n, 4100 + n)
    dd, de = torch.from_numpy(d).cuda(), torch.from_numpy(np.append(e, 0.0)).cuda()
    z = torch.full((n, n), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    status = np.zeros(4, np.int32)
    assert helpers.run_stedc(n, *[ctypes.c_void_p(v.data_ptr()) for v in (dd, de, z)], n, m_cols, 16, code,
                             status.ctypes.data_as(ctypes.c_void_p)) == 0
    return d, e, dd.cpu().numpy(), z.cpu().numpy().T, status[0]


@pytest.mark.parametrize("n,m_cols", [(5, 1), (9, 8), (40, 3), (64, 63), (100, 30)])
def test_stedc_writes_only_the_wanted_vectors(helpers, n, m_cols):
    d, e, w, z, code = _stedc(helpers, n, m_cols, 0)
    assert code == 0
    t = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    np.testing.assert_allclose(w, np.linalg.eigvalsh(t), rtol=0, atol=5e-14 * n)
    assert np.abs(t @ z[:, :m_cols] - z[:, :m_cols] * w[:m_cols]).max() < 1e-13 * n
    assert np.all(z[:, m_cols:] == 7.0)


@pytest.mark.parametrize("n", [5, 40, 64])
def test_stedc_after_a_failed_stage(helpers, n):
    """One subtree is the whole solve: after an error of an earlier stage it leaves its inputs and outputs alone."""
    d, _, w, z, code = _stedc(helpers, n, n, 3)
    assert code == 3 and np.array_equal(w, d) and np.all(z == 7.0)
