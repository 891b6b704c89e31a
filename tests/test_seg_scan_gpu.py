"""What the host reads after the scan of the row-segment counts, before it uses
them: the totals, the status word (a gradient tile that gave up has left its
counts unwritten) and whether the scan itself gave up."""

import ctypes
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "seg_scan_device.cu")
OUT = os.path.join(ROOT, "tests", "_build", "seg_scan_device.so")
CSRC = os.path.join(ROOT, "dmsc_b200", "csrc")
DEPS = [SRC, os.path.join(CSRC, "scan.cuh"), os.path.join(CSRC, "common.cuh")]
LOOKS = 1 << 20


@pytest.fixture(scope="module")
def lib():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    nvcc = cand if os.path.exists(cand) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc not available")
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-Xcompiler",
                               "-fPIC", "-shared", "--expt-relaxed-constexpr", "-o", OUT + ".tmp", SRC])
        os.replace(OUT + ".tmp", OUT)
    lib = ctypes.CDLL(OUT)
    lib.seg_scan_device.argtypes = [ctypes.c_longlong, ctypes.c_uint, ctypes.c_int, ctypes.c_void_p]
    return lib


def _words(lib, n, status, looks):
    w = (ctypes.c_longlong * 5)()
    assert lib.seg_scan_device(n, status, looks, w) == 0
    return list(w)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 300_001])
@pytest.mark.parametrize("status", [0, 64])
def test_totals_and_status(lib, n, status):
    assert _words(lib, n, status, LOOKS) == [n, 2 * n, 3 * n, status, 0]


@pytest.mark.parametrize("n,gives_up", [(4096, 0), (4097, 2), (300_001, 2)])
def test_scan_without_looks(lib, n, gives_up):
    assert _words(lib, n, 0, 0)[4] == gives_up
