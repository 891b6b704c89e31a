"""Rows by multiplication: row_magic and row_of of csrc/common.cuh, compiled for
the host, against the integer division, at the indices where they could be off
by one. CPU only; needs nvcc."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "row_of_host.cu")
OUT = os.path.join(ROOT, "tests", "_build", "row_of_host.so")
DEPS = [SRC, os.path.join(ROOT, "dmsc_b200", "csrc", "common.cuh")]
CELLS = 1 << 29  # an image's indices stay below: four cell ids an index


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
    lib.row_of_host.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 2 + [ctypes.c_int] + [ctypes.c_void_p] * 2
    return lib


def _widths():
    rng = np.random.default_rng(5)
    near = [(1 << k) + d for k in range(1, 29) for d in (-1, 0, 1)]
    return sorted({n for n in near + [int(2 ** e) for e in rng.uniform(1, 28.99, 300)] if 2 <= n < CELLS // 2})


@pytest.mark.parametrize("part", range(4))
def test_rows_are_quotients(lib, part):
    rng = np.random.default_rng(part)
    magic, shift = ctypes.c_uint(), ctypes.c_int()
    for nx in _widths()[part::4]:
        top = (CELLS - 1) // nx
        q = np.concatenate([[0, 1, top - 1, top], rng.integers(0, top + 1, 60)]).astype(np.int64)
        l = (q[:, None] * nx + np.array([-1, 0, 1, nx - 2, nx - 1])).ravel()
        l = np.concatenate([l, [CELLS - 1]])
        l = np.ascontiguousarray(l[(l >= 0) & (l < CELLS)].astype(np.int32))
        row = np.empty_like(l)
        lib.row_of_host(nx, l.ctypes.data, row.ctypes.data, l.size, ctypes.byref(magic), ctypes.byref(shift))
        assert magic.value < 1 << 30, nx  # so that the product stays below 2^59
        assert np.array_equal(row, l // nx), nx
