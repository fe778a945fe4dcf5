"""The plans of the resident reduction for devices with fewer SMs (a partition of a GPU), on the CPU: the library's own
planning functions are called through their exported names.

Option "sytrd_grid" takes any number of CTAs, however many rows each then owns.  The no-allocation entry takes every n up
to 1792 whose rows the device holds on chip.  Rows per CTA, and with them the kernel a plan selects, depend on the number
of SMs.
"""
import ctypes
import re
import subprocess

import pytest

import xtbeig

MAX_SMEM = 232448 - 2048  # what the entry passes for a B200


class Plan(ctypes.Structure):
    _fields_ = [(f, ctypes.c_int) for f in ("grid", "threads", "cpt", "reg_rows", "rows_per_cta", "ldr")] + [
        ("rows_in_smem", ctypes.c_bool), ("supported", ctypes.c_bool), ("smem", ctypes.c_size_t)]


@pytest.fixture(scope="module")
def functions():
    out = subprocess.run(["nm", "-D", "--defined-only", xtbeig.LIB_PATH], capture_output=True, text=True).stdout
    name = lambda what: re.search(r"\b(\w*%s\w*)$" % what, out, flags=re.M).group(1)
    lib = ctypes.CDLL(xtbeig.LIB_PATH)
    plan = getattr(lib, name("sytrd_planIdE"))
    plan.argtypes, plan.restype = [ctypes.c_int, ctypes.c_int, ctypes.c_size_t, ctypes.c_int], Plan
    supported = getattr(lib, name("sytrd_upper_inplace_supported"))
    supported.argtypes, supported.restype = [ctypes.POINTER(Plan)], ctypes.c_bool
    return plan, supported


@pytest.mark.parametrize("sms", [148, 132, 74, 36, 18, 9])
def test_every_plan_on_chip_has_a_kernel(functions, sms):
    plan, supported = functions
    for n in range(1, 1793):
        pl = plan(n, sms, MAX_SMEM, 0)
        # The rows of the matrix in shared memory alone fit: then the call is not refused.
        rows = -(-n // max(1, min(sms, (n + 3) // 4)))
        if (rows + 1) * (n + n % 2) * 8 + 16384 <= MAX_SMEM:
            assert pl.rows_in_smem, (n, sms)
        if pl.rows_in_smem:
            assert pl.supported and supported(ctypes.byref(pl)), (n, sms)


@pytest.mark.parametrize("n", [1, 63, 500, 1788, 2049, 4096, 4097, 8192, 8193, 16384])
def test_a_chosen_grid_fits_in_shared_memory(functions, n):
    plan, _ = functions
    for grid in range(1, 149):
        pl = plan(n, 148, MAX_SMEM, grid)
        assert pl.supported and pl.smem <= MAX_SMEM and grid <= pl.grid <= 148, grid
        if n <= 1024 or grid >= 64:
            assert pl.grid == grid
